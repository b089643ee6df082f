// swm_ops.cu -- FP64 geometry precompute, per-operator (unfused) FP64
// kernels, cube-edge syncs on fields, state combinations and deterministic
// FP64 reductions.
#include "swm_ops.cuh"
#include "swm_stage.cuh"

namespace swm {

namespace {

constexpr double kPi = 3.141592653589793238462643383279502884;

// Panel frames (ex, ey, inward normal n) of the six cube faces
// (topology/cubed_sphere_topology_mod.f90:29-55 of the reference).
__constant__ int c_ex[6][3] = {{-1, 0, 0}, {0, 0, -1}, {1, 0, 0}, {0, 0, 1}, {1, 0, 0}, {1, 0, 0}};
__constant__ int c_ey[6][3] = {{0, 1, 0}, {0, 1, 0}, {0, 1, 0}, {0, 1, 0}, {0, 0, 1}, {0, 0, -1}};
__constant__ int c_n[6][3] = {{0, 0, 1}, {-1, 0, 0}, {0, 0, -1}, {1, 0, 0}, {0, 1, 0}, {0, -1, 0}};

constexpr int TPB = 256;

inline int nblk(long long count, int tpb = TPB) { return (int)((count + tpb - 1) / tpb); }

// valid node g in [0, 6n^2) -> (p, i, j, pitched index)
struct NodeIx {
  int p, i, j;
  long long idx;
};
__device__ __forceinline__ NodeIx node_of(const FieldGeom& g, long long gi) {
  NodeIx r;
  const long long nn = (long long)g.n * g.n;
  r.p = (int)(gi / nn);
  const long long rem = gi - (long long)r.p * nn;
  r.j = (int)(rem / g.n);
  r.i = (int)(rem - (long long)r.j * g.n);
  r.idx = (long long)r.p * g.ps + (long long)r.j * g.P + r.i;
  return r;
}

// ---------------------------------------------------------------------------
// Geometry: equiangular cubed sphere metric on the unit sphere
// (equiang_cs/ecs_metric_mod.f90:326-478, mesh_factory_mod.f90:85-133,
// coriolis_factory_mod.f90:151-172).  alpha_i = -pi/4 + i*hx, hx = (pi/2)/N.
// ---------------------------------------------------------------------------
__global__ void geometry_kernel(FieldGeom g, double hx, double radius, double omega, double ax,
                                double ay, double az, double* m) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const NodeIx k = node_of(g, gi);
  const double al = -0.25 * kPi + k.i * hx, be = -0.25 * kPi + k.j * hx;
  const double ta = tan(al), tb = tan(be);
  const double sg = sqrt(1.0 + ta * ta + tb * tb);
  const double A = 1.0 + ta * ta, B = 1.0 + tb * tb;
  const double J = A * B / (sg * sg * sg);
  m[MJ * g.fs + k.idx] = J;
  m[MQI1 * g.fs + k.idx] = sg * sg / A;
  m[MQI2 * g.fs + k.idx] = sg * sg * ta * tb / (A * B);
  m[MQI3 * g.fs + k.idx] = sg * sg / B;
  // point on the sphere: proto-face (ta, tb, 1)/sg mapped to panel p
  const double rp[3] = {ta / sg, tb / sg, 1.0 / sg};
  double r[3];
  for (int c = 0; c < 3; ++c)
    r[c] = c_ex[k.p][c] * rp[0] + c_ey[k.p][c] * rp[1] - c_n[k.p][c] * rp[2];
  const double nn = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
  m[MF * g.fs + k.idx] = 2.0 * omega * ((ax * r[0] + ay * r[1] + az * r[2]) / nn);
  m[MRJ * g.fs + k.idx] = 1.0 / (J * hx * radius);
}

__device__ void a1p(double a, double b, double v[3]) {
  const double ta = tan(a), tb = tan(b);
  const double p = pow(1.0 + ta * ta + tb * tb, 1.5);
  v[0] = (1.0 + ta * ta) * (1.0 + tb * tb) / p;
  v[1] = -ta * tb * (1.0 + ta * ta) / p;
  v[2] = -ta * (1.0 + ta * ta) / p;
}
__device__ void a2p(double a, double b, double v[3]) {
  const double ta = tan(a), tb = tan(b);
  const double p = pow(1.0 + ta * ta + tb * tb, 1.5);
  v[0] = -ta * tb * (1.0 + tb * tb) / p;
  v[1] = (1.0 + ta * ta) * (1.0 + tb * tb) / p;
  v[2] = -tb * (1.0 + tb * tb) / p;
}
__device__ void b1p(double a, double b, double v[3]) {
  const double ta = tan(a), tb = tan(b);
  const double s = sqrt(1.0 + ta * ta + tb * tb);
  v[0] = (1.0 + tb * tb - (ta * tb) * (ta * tb) / (1.0 + ta * ta)) / s;
  v[1] = 0.0;
  v[2] = -ta * (1.0 + tb * tb / (1.0 + ta * ta)) / s;
}
__device__ void b2p(double a, double b, double v[3]) {
  const double ta = tan(a), tb = tan(b);
  const double s = sqrt(1.0 + ta * ta + tb * tb);
  v[0] = 0.0;
  v[1] = ((1.0 + ta * ta) - (ta * tb) * (ta * tb) / (1.0 + tb * tb)) / s;
  v[2] = -tb * (ta * ta / (1.0 + tb * tb) + 1.0) / s;
}

// Cartesian contravariant basis vectors b1, b2 of every node, mapped from
// the prototype face to panel p (mesh_factory_mod.f90:131-132 with
// ecs_metric_mod.f90 calculate_b1/b2): 6 fields b1x b1y b1z b2x b2y b2z.
__global__ void basis_kernel(FieldGeom g, double hx, double* b) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const NodeIx k = node_of(g, gi);
  const double al = -0.25 * kPi + k.i * hx, be = -0.25 * kPi + k.j * hx;
  double v1[3], v2[3];
  b1p(al, be, v1);
  b2p(al, be, v2);
  for (int c = 0; c < 3; ++c) {
    b[c * g.fs + k.idx] = c_ex[k.p][c] * v1[0] + c_ey[k.p][c] * v1[1] - c_n[k.p][c] * v1[2];
    b[(3 + c) * g.fs + k.idx] = c_ex[k.p][c] * v2[0] + c_ey[k.p][c] * v2[1] - c_n[k.p][c] * v2[2];
  }
}

// Covariant-vector sync weights: dot products of the basis vectors of the
// two panels across each edge (ecs_Ah_vec_sync_factory_mod.f90:97-144).
__global__ void sync_weights_kernel(int n, double hx, double* qw) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double c = -0.25 * kPi + k * hx, q = 0.25 * kPi;
  double a[3], b[3];
  a2p(c, -q, a); b1p(c, q, b);
  qw[k] = a[0] * b[0] + a[1] * (-b[2]) + a[2] * b[1];
  a2p(c, q, a); b1p(c, -q, b);
  qw[n + k] = a[0] * b[0] + a[1] * b[2] + a[2] * (-b[1]);
  a1p(-q, c, a); b2p(q, c, b);
  qw[2 * n + k] = a[0] * (-b[2]) + a[1] * b[1] + a[2] * b[0];
  a1p(q, c, a); b2p(-q, c, b);
  qw[3 * n + k] = a[0] * b[2] + a[1] * b[1] + a[2] * (-b[0]);
}

__global__ void to_f32_kernel(const double* s, float* d, long long count) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) d[k] = (float)s[k];
}

// ---------------------------------------------------------------------------
// Per-operator FP64 kernels (reference formulas and operation order).
// ---------------------------------------------------------------------------
__global__ void co2contra_kernel(FieldGeom g, const double* m, const double* u, const double* v,
                                 double* ut, double* vt) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const long long x = node_of(g, gi).idx;
  const double q1 = m[MQI1 * g.fs + x], q2 = m[MQI2 * g.fs + x], q3 = m[MQI3 * g.fs + x];
  const double a = q1 * u[x] + q2 * v[x];
  const double b = q2 * u[x] + q3 * v[x];
  ut[x] = a;
  vt[x] = b;
}

__global__ void massflux_kernel(FieldGeom g, const double* h, const double* ut, const double* vt,
                                double* hu, double* hv) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const long long x = node_of(g, gi).idx;
  hu[x] = 1.0 * h[x] * ut[x];
  hv[x] = 1.0 * h[x] * vt[x];
}

__global__ void ke_kernel(FieldGeom g, const double* u, const double* v, const double* ut,
                          const double* vt, double* ke) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const long long x = node_of(g, gi).idx;
  ke[x] = (u[x] * ut[x] + v[x] * vt[x]) / 2.0;
}

__global__ void ke_update_kernel(FieldGeom g, double grav, const double* h, const double* hs,
                                 double* ke) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const long long x = node_of(g, gi).idx;
  ke[x] = ke[x] + grav * h[x] + grav * (hs ? hs[x] : 0.0);
}

// Differential operators with their cube-edge syncs in one launch, on the
// node ranges of the FP64 stage kernel (swm_stage.cuh): straight-line interior,
// closure columns in warps of their own, and a boundary node's own and
// neighbour terms formed by two lanes.  FP64 bounds the interior and latency
// the small panels; as a pass over table-driven stencils (the curl with the
// reference's J (v / J), two divisions a tap) and two sync launches, the curl
// at N=130 took 61 us a call with its synchronisation, the divergence 34 and the
// gradient 30; each now 25.
struct OpArgs {
  FieldGeom g;
  const double *a, *b, *m, *qw;   // a, b: input fields (grad: a)
  double s;                        // grad: 1 / (hx a)
  double *o1, *o2;
};

// The copies of a boundary node: raw(p, i, j, L) is called for the node itself
// (even lane, L null) and for the neighbours' nodes at the same point (odd
// lane, L the link that led there and slr whether it crosses a left / right
// side); its results x, y add up over the copies of both lanes.
template <class F>
__device__ __forceinline__ void over_copies(const Topology& tp, int n, int tid, const PointAt& at, F raw,
                                            double& x, double& y) {
  const int e = n - 1, i = at.i, j = at.j;
  const bool lr = (i == 0) | (i == e), bt = (j == 0) | (j == e), own = (tid & 1) == 0;
  x = y = 0.0;
  const int copies = !own && lr && bt ? 2 : 1;
#pragma unroll 1
  for (int s = 0; s < copies; ++s) {
    const bool slr = lr && s == 0;
    int q = at.p, iq = i, jq = j;
    EdgeLink L{};
    if (!own) {
      L = tp.link[at.p][slr ? (i == 0 ? SIDE_L : SIDE_R) : (j == 0 ? SIDE_B : SIDE_T)];
      const int k = slr ? j : i, kk = L.rev ? e - k : k;
      q = L.q;
      iq = L.side_q == SIDE_L ? 0 : L.side_q == SIDE_R ? e : kk;
      jq = L.side_q == SIDE_B ? 0 : L.side_q == SIDE_T ? e : kk;
    }
    double a, b;
    raw(q, iq, jq, own ? nullptr : &L, slr, a, b);
    x += a;
    y += b;
  }
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  y += __shfl_xor_sync(0xffffffffu, y, 1);
}
__device__ __forceinline__ double copy_weight(int n, const PointAt& at) {
  const bool lr = (at.i == 0) | (at.i == n - 1), bt = (at.j == 0) | (at.j == n - 1);
  return lr && bt ? 1.0 / 3.0 : 0.5;
}

// grad_ah_sbp_t%calc_grad (grad_ah_sbp_mod.f90:26-90) with its covariant sync
// (ecs_Ah_vec_sync_mod.f90:62-125)
template <int ORD>
__global__ void __launch_bounds__(PT_TPB)
    grad_kernel(const __grid_constant__ OpArgs a, const __grid_constant__ Topology tp) {
  constexpr int NE = Ord<ORD>::NE;
  const FieldGeom& g = a.g;
  const int n = g.n, P = g.P, tid = blockIdx.x * PT_TPB + threadIdx.x;
  PointAt at;
  if (!point_at<ORD>(n, tid, at)) return;
  const int i = at.i, j = at.j;
  const long long x = (long long)at.p * g.ps + (long long)j * P + i;
  auto raw = [&](int p, int ii, int jj, double& gx, double& gy) {
    const double* f = a.a + (long long)p * g.ps + (long long)jj * P + ii;
    gx = a.s * taps_sum<ORD>(taps_of<ORD>(ii, n), f, ii, 1);
    gy = a.s * taps_sum<ORD>(taps_of<ORD>(jj, n), f, jj, P);
  };
  double gx, gy;
  if (at.boundary) {
    over_copies(tp, n, tid, at, [&](int p, int ii, int jj, const EdgeLink* L, bool slr, double& ax, double& ay) {
      raw(p, ii, jj, ax, ay);
      if (!L) return;
      const double rx = L->dim_i ? L->istep * ax : L->jstep * ay;
      const double ry = L->dim_i ? L->jstep * ay : L->istep * ax;
      ax = slr ? rx + a.qw[(i == 0 ? 2 : 3) * n + j] * ry : rx;
      ay = slr ? ry : ry + a.qw[(j == 0 ? 0 : 1) * n + i] * rx;
    }, gx, gy);
    if ((tid & 1) || !at.live) return;
    const double w = copy_weight(n, at);
    gx *= w;
    gy *= w;
  } else if (i >= NE && i < n - NE && j >= NE && j < n - NE) {
    const double* f = a.a + x;
    const double c = a.s * d_coef<ORD>(1);
    gx = c * d_ratio<ORD, double>([&](int o) { return f[o] - f[-o]; });
    gy = c * d_ratio<ORD, double>([&](int o) { return f[o * P] - f[-o * P]; });
  } else {
    raw(at.p, i, j, gx, gy);
  }
  a.o1[x] = gx;
  a.o2[x] = gy;
}

// Pre-sync curl (Dx b - Dy a) / (J hx a) of the covariant (a, b), or
// divergence (Dx(J a) + Dy(J b)) / (J hx a) of the contravariant ones, at any
// node.
template <int ORD, bool CURL>
__device__ __forceinline__ double div_raw(const OpArgs& A, int p, int i, int j) {
  const FieldGeom& g = A.g;
  const int n = g.n, P = g.P;
  const long long x = (long long)p * g.ps + (long long)j * P + i;
  const Taps<ORD> tx = taps_of<ORD>(i, n), ty = taps_of<ORD>(j, n);
  double s;
  if (CURL) {
    s = taps_sum<ORD>(tx, A.b + x, i, 1) - taps_sum<ORD>(ty, A.a + x, j, P);
  } else {
    const double* J = A.m + MJ * g.fs + x;
    s = 0.0;
#pragma unroll
    for (int k = 0; k < Taps<ORD>::NT; ++k) {
      const int ox = tx.s + k - i, oy = (ty.s + k - j) * P;
      s += tx.c[k] * (J[ox] * (tx.has(k) ? A.a[x + ox] : 0.0));
      s += ty.c[k] * (J[oy] * (ty.has(k) ? A.b[x + oy] : 0.0));
    }
  }
  return s * A.m[MRJ * g.fs + x];
}
// The synced value at a node; live false for lanes that store nothing.
template <int ORD, bool CURL>
__device__ __forceinline__ double div_synced(const OpArgs& A, const Topology& tp, int tid, const PointAt& at,
                                             bool& live) {
  constexpr int NE = Ord<ORD>::NE;
  const FieldGeom& g = A.g;
  const int n = g.n, P = g.P, i = at.i, j = at.j;
  live = true;
  if (at.boundary) {
    double d, unused;
    over_copies(tp, n, tid, at, [&](int p, int ii, int jj, const EdgeLink*, bool, double& v, double& w) {
      v = div_raw<ORD, CURL>(A, p, ii, jj);
      w = 0.0;
    }, d, unused);
    live = !(tid & 1) && at.live;
    return d * copy_weight(n, at);
  }
  if (!(i >= NE && i < n - NE && j >= NE && j < n - NE)) return div_raw<ORD, CURL>(A, at.p, i, j);
  const long long x = (long long)at.p * g.ps + (long long)j * P + i;
  const double *U = A.a + x, *V = A.b + x, *J = A.m + MJ * g.fs + x;
  const double rJ = A.m[MRJ * g.fs + x] * d_coef<ORD>(1);
  if (CURL)
    return rJ * d_ratio<ORD, double>([&](int o) { return (V[o] - V[-o]) - (U[o * P] - U[-o * P]); });
  return rJ * d_ratio<ORD, double>([&](int o) {
           return (J[o] * U[o] - J[-o] * U[-o]) + (J[o * P] * V[o * P] - J[-o * P] * V[-o * P]);
         });
}

// curl_div_based_t%calc_curl (curl_div_based_mod.f90:26-66) and
// div_ah_sbp_t%calc_div (div_ah_sbp_mod.f90:24-98), synced
template <int ORD, bool CURL>
__global__ void __launch_bounds__(PT_TPB)
    div_kernel(const __grid_constant__ OpArgs a, const __grid_constant__ Topology tp) {
  const int tid = blockIdx.x * PT_TPB + threadIdx.x;
  PointAt at;
  if (!point_at<ORD>(a.g.n, tid, at)) return;
  bool live;
  const double d = div_synced<ORD, CURL>(a, tp, tid, at, live);
  if (live) a.o1[(long long)at.p * a.g.ps + (long long)at.j * a.g.P + at.i] = d;
}

__global__ void coriolis_kernel(FieldGeom g, const double* m, const double* hu, const double* hv,
                                const double* h, const double* cu, double* cor_u, double* cor_v) {
  const long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6LL * g.n * g.n) return;
  const long long x = node_of(g, gi).idx;
  const double fz = m[MF * g.fs + x] + cu[x];
  const double J = m[MJ * g.fs + x];
  cor_u[x] = fz * hv[x] / h[x] * J;
  cor_v[x] = -(fz * hu[x] / h[x] * J);
}

__global__ void fill_kernel(long long count, double value, double* out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) out[k] = value;
}

__global__ void axpby_kernel(long long count, double s1, const double* a, double s2,
                             const double* b, double* out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  out[k] = b ? s1 * a[k] + s2 * b[k] : s1 * a[k];
}

// gather boundary values of up to two fields into edge slots v0 (and v1)
template <class T>
__global__ void gather_edge_kernel(FieldGeom g, const T* f0, int v0, const T* f1, int v1, T* E) {
  const int n = g.n, nb = 4 * n - 4;
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6 * nb) return;
  const int p = gi / nb;
  int i, j;
  boundary_node(gi - p * nb, n, i, j);
  const long long x = (long long)p * g.ps + (long long)j * g.P + i;
  const T a = f0[x], b = f1 ? f1[x] : T(0);
  auto put = [&](int side, int k) {
    E[((long long)(p * 4 + side) * 4 + v0) * n + k] = a;
    if (f1) E[((long long)(p * 4 + side) * 4 + v1) * n + k] = b;
  };
  if (i == 0) put(SIDE_L, j);
  if (i == n - 1) put(SIDE_R, j);
  if (j == 0) put(SIDE_B, i);
  if (j == n - 1) put(SIDE_T, i);
}

template <class T>
__global__ void sync_scalar_kernel(FieldGeom g, Topology tp, const T* E, T* f) {
  const int n = g.n, nb = 4 * n - 4;
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6 * nb) return;
  const int p = gi / nb;
  int i, j;
  boundary_node(gi - p * nb, n, i, j);
  const long long x = (long long)p * g.ps + (long long)j * g.P + i;
  const EdgeView<T> ev{E, n};
  f[x] = sync_scalar_node<T>(ev, tp, p, i, j, EV_ZETA, f[x]);
}

template <class T>
__global__ void sync_vector_kernel(FieldGeom g, Topology tp, const double* qw, const T* E, T* gx,
                                   T* gy) {
  const int n = g.n, nb = 4 * n - 4;
  const int gi = blockIdx.x * blockDim.x + threadIdx.x;
  if (gi >= 6 * nb) return;
  const int p = gi / nb;
  int i, j;
  boundary_node(gi - p * nb, n, i, j);
  const long long x = (long long)p * g.ps + (long long)j * g.P + i;
  const EdgeView<T> ev{E, n};
  T a = gx[x], b = gy[x];
  sync_vector_node<T>(ev, tp, qw, p, i, j, a, b);
  gx[x] = a;
  gy[x] = b;
}

// ---------------------------------------------------------------------------
// Deterministic reductions: fixed grid, per-block tree, then one block sums
// the partials in a fixed order.
// ---------------------------------------------------------------------------
__global__ void reduce_partial_kernel(FieldGeom g, int kind, const double* a, const double* b,
                                      const double* J, const double* Aw, double hx2,
                                      double* partial) {
  __shared__ double sh[TPB];
  const long long total = 6LL * g.n * g.n;
  double acc = 0.0;
  for (long long gi = (long long)blockIdx.x * blockDim.x + threadIdx.x; gi < total;
       gi += (long long)gridDim.x * blockDim.x) {
    const NodeIx k = node_of(g, gi);
    double val = a[k.idx];
    if (kind == 0 && b) val = val * b[k.idx];
    if (kind == 1) val = val * J[k.idx] * hx2 * Aw[k.i] * Aw[k.j];
    acc += val;
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = TPB / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void reduce_final_kernel(const double* partial, int np, double* result) {
  __shared__ double sh[TPB];
  double acc = 0.0;
  for (int k = threadIdx.x; k < np; k += blockDim.x) acc += partial[k];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = TPB / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) *result = sh[0];
}

// The seven global values of get_diagnostics (operator_swm_mod.f90:115-155) in
// one pass: minimum and maximum of h, and the SBP integrals of h, of the kinetic
// and potential energy and of the enstrophy, with the synced curl formed where
// it is used.  Per-block trees, then one block over the partials in a fixed
// order: two launches instead of 19 (curl, syncs, integrands and a pair of
// launches per value), 158 -> 66 us a call at N=130.
constexpr int DIAG_N = 6;   // hmin, hmax, mass, KE, PE, enstrophy

__device__ __forceinline__ double diag_op(int k, double x, double y) {
  return k == 0 ? fmin(x, y) : k == 1 ? fmax(x, y) : x + y;
}

template <int ORD>
__global__ void __launch_bounds__(PT_TPB, DIAG_BLOCKS / 152)   // its grid is one wave
    diag_kernel(const __grid_constant__ OpArgs a, const __grid_constant__ Topology tp, const double* h,
                const double* hs, const double* Aw, double grav, double hx2, int threads, double* partial) {
  const FieldGeom& g = a.g;
  const int n = g.n;
  const long long fs = g.fs;
  double r[DIAG_N] = {INFINITY, -INFINITY, 0.0, 0.0, 0.0, 0.0};
  // whole blocks of nodes a turn, so that the lanes of a pair stay together
  for (int t0 = blockIdx.x * PT_TPB; t0 < threads; t0 += gridDim.x * PT_TPB) {
    PointAt at;
    const int tid = t0 + threadIdx.x;
    if (!point_at<ORD>(n, tid, at)) continue;
    bool live;
    const double z = div_synced<ORD, true>(a, tp, tid, at, live);
    if (!live) continue;
    const long long x = (long long)at.p * g.ps + (long long)at.j * g.P + at.i;
    const double u = a.a[x], v = a.b[x], hh = h[x], q2 = a.m[MQI2 * fs + x];
    const double ut = a.m[MQI1 * fs + x] * u + q2 * v, vt = q2 * u + a.m[MQI3 * fs + x] * v;
    const double w = a.m[MJ * fs + x] * hx2 * Aw[at.i] * Aw[at.j];
    const double ph = hs ? hh + hs[x] : hh, c = z + a.m[MF * fs + x];
    r[0] = fmin(r[0], hh);
    r[1] = fmax(r[1], hh);
    r[2] += hh * w;
    r[3] += (0.5 * hh * (ut * u + vt * v)) * w;
    r[4] += (0.5 * grav * ph * ph) * w;
    r[5] += (0.5 * c * c / hh) * w;
  }
  __shared__ double sh[DIAG_N][PT_TPB / 32];
#pragma unroll
  for (int k = 0; k < DIAG_N; ++k) {
    for (int o = 16; o > 0; o >>= 1) r[k] = diag_op(k, r[k], __shfl_xor_sync(0xffffffffu, r[k], o));
    if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = r[k];
  }
  __syncthreads();
  if (threadIdx.x < DIAG_N) {
    double s = sh[threadIdx.x][0];
    for (int t = 1; t < PT_TPB / 32; ++t) s = diag_op(threadIdx.x, s, sh[threadIdx.x][t]);
    partial[threadIdx.x * gridDim.x + blockIdx.x] = s;
  }
}

// one warp per value
__global__ void diag_final_kernel(const double* partial, int np, double* result) {
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = k == 0 ? INFINITY : k == 1 ? -INFINITY : 0.0;
  for (int t = lane; t < np; t += 32) s = diag_op(k, s, partial[k * np + t]);
  for (int o = 16; o > 0; o >>= 1) s = diag_op(k, s, __shfl_xor_sync(0xffffffffu, s, o));
  if (lane == 0) result[k] = s;
}

// ---------------------------------------------------------------------------
// FP32 (hi, lo) pair helpers
// ---------------------------------------------------------------------------
// FP32 (hi, lo) pairs combined in double-float arithmetic: error-free
// two-sum and two-product (fmaf), then renormalisation; the coefficients
// come split into float pairs.  FP32 instructions only (GB300's FP64 rate
// would bound an FP64 evaluation); about 2^-44 relative accuracy.
__device__ __forceinline__ void quick_two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  e = b - (s - a);
}
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ __forceinline__ void df_mul(float xh, float xl, float yh, float yl, float& h, float& l) {
  const float p = xh * yh;
  float e = fmaf(xh, yh, -p);
  e = fmaf(xh, yl, e);
  e = fmaf(xl, yh, e);
  quick_two_sum(p, e, h, l);
}
__device__ __forceinline__ void df_add(float ah, float al, float bh, float bl, float& h, float& l) {
  float sm, e;
  two_sum(ah, bh, sm, e);
  e += al + bl;
  quick_two_sum(sm, e, h, l);
}

__global__ void axpby_pair_kernel(long long count, float s1h, float s1l, const float* ahi,
                                  const float* alo, float s2h, float s2l, const float* bhi,
                                  const float* blo, float* ohi, float* olo) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  float h, l;
  df_mul(s1h, s1l, ahi[k], alo[k], h, l);
  if (bhi) {
    float h2, l2;
    df_mul(s2h, s2l, bhi[k], blo[k], h2, l2);
    df_add(h, l, h2, l2, h, l);
  }
  ohi[k] = h;
  olo[k] = l;
}

__global__ void fill_pair_kernel(long long count, float vh, float vl, float* ohi, float* olo) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  ohi[k] = vh;
  olo[k] = vl;
}

__global__ void split_kernel(long long count, const double* s, float* hi, float* lo) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const float h = (float)s[k];
  hi[k] = h;
  lo[k] = (float)(s[k] - (double)h);
}

__global__ void join_kernel(long long count, const float* hi, const float* lo, double* d) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  d[k] = (double)hi[k] + (double)lo[k];
}

// Packed <-> pitched state fields.  Thread k handles packed value k of the
// nf fields (k = c*6*n*n + (p*n + j)*n + i), so a warp touches 32
// consecutive packed doubles: whole 128-byte lines of the packed side, which
// may sit in host memory behind the host-device link.  The state fields hold
// n*P pitched rows per panel (ps = n*P).  Indices fit 32 bits for n <= 8191.
__device__ __forceinline__ void packed_index(const FieldGeom& g, unsigned k, unsigned& c,
                                             unsigned& r, long long& o) {
  const unsigned n = (unsigned)g.n, nn6 = 6u * n * n;
  c = k / nn6;
  r = k - c * nn6;
  const unsigned row = r / n;
  o = (long long)c * g.fs + (long long)row * g.P + (r - row * n);
}

__device__ __forceinline__ double* field_of(const PackedFields& pf, unsigned c) {
  return c == 0 ? pf.f[0] : (c == 1 ? pf.f[1] : pf.f[2]);
}

template <class T>
__global__ void unpack_kernel(FieldGeom g, unsigned total, PackedFields src, T* hi, float* lo) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= total) return;
  unsigned c, r;
  long long o;
  packed_index(g, k, c, r, o);
  const double x = field_of(src, c)[r];
  if constexpr (sizeof(T) == 8) {
    hi[o] = x;
  } else {
    const float h = (float)x;
    hi[o] = h;
    lo[o] = (float)(x - (double)h);
  }
}

template <class T>
__global__ void pack_kernel(FieldGeom g, unsigned total, const T* hi, const float* lo,
                            PackedFields dst) {
  const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= total) return;
  unsigned c, r;
  long long o;
  packed_index(g, k, c, r, o);
  double x;
  if constexpr (sizeof(T) == 8) x = hi[o];
  else x = (double)hi[o] + (double)lo[o];
  field_of(dst, c)[r] = x;
}

}  // namespace

// ===========================================================================
// launchers
// ===========================================================================
cudaError_t launch_geometry(const FieldGeom& g, int N, double radius, double omega,
                            const double axis[3], double* m64, double* qw, cudaStream_t st) {
  const double hx = (0.25 * kPi - (-0.25 * kPi)) / (double)N;
  const double an = sqrt(axis[0] * axis[0] + axis[1] * axis[1] + axis[2] * axis[2]);
  geometry_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, hx, radius, omega, axis[0] / an,
                                                          axis[1] / an, axis[2] / an, m64);
  sync_weights_kernel<<<nblk(g.n), TPB, 0, st>>>(g.n, hx, qw);
  return cudaGetLastError();
}

cudaError_t launch_basis(const FieldGeom& g, double hx, double* b, cudaStream_t st) {
  basis_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, hx, b);
  return cudaGetLastError();
}

cudaError_t launch_to_f32(const double* src, float* dst, long long count, cudaStream_t st) {
  to_f32_kernel<<<nblk(count), TPB, 0, st>>>(src, dst, count);
  return cudaGetLastError();
}

cudaError_t launch_co2contra(const FieldGeom& g, const double* m64, const double* u,
                             const double* v, double* ut, double* vt, cudaStream_t st) {
  co2contra_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, m64, u, v, ut, vt);
  return cudaGetLastError();
}

cudaError_t launch_massflux(const FieldGeom& g, const double* h, const double* ut,
                            const double* vt, double* hu, double* hv, cudaStream_t st) {
  massflux_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, h, ut, vt, hu, hv);
  return cudaGetLastError();
}

cudaError_t launch_ke(const FieldGeom& g, const double* u, const double* v, const double* ut,
                      const double* vt, double* ke, cudaStream_t st) {
  ke_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, u, v, ut, vt, ke);
  return cudaGetLastError();
}

cudaError_t launch_ke_update(const FieldGeom& g, double grav, const double* h, const double* hs,
                             double* ke, cudaStream_t st) {
  ke_update_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, grav, h, hs, ke);
  return cudaGetLastError();
}

#define SWM_BY_ORDER(order, call)                  \
  switch (order) {                                 \
    case 21: { constexpr int ORD = 21; call; } break; \
    case 42: { constexpr int ORD = 42; call; } break; \
    case 43: { constexpr int ORD = 43; call; } break; \
    case 63: { constexpr int ORD = 63; call; } break; \
    default: return cudaErrorInvalidValue;         \
  }

cudaError_t launch_grad(const FieldGeom& g, int order, const Topology& tp, const double* qw, double ghs,
                        const double* f, double* gx, double* gy, cudaStream_t st) {
  const OpArgs a{g, f, nullptr, nullptr, qw, ghs, gx, gy};
  SWM_BY_ORDER(order, (grad_kernel<ORD><<<point_ranges<ORD>(g.n).total / PT_TPB, PT_TPB, 0, st>>>(a, tp)));
  return cudaGetLastError();
}

cudaError_t launch_div(const FieldGeom& g, int order, const Topology& tp, const double* m64, const double* u,
                       const double* v, bool curl, double* out, cudaStream_t st) {
  const OpArgs a{g, u, v, m64, nullptr, 0.0, out, nullptr};
  if (curl) {
    SWM_BY_ORDER(order, (div_kernel<ORD, true><<<point_ranges<ORD>(g.n).total / PT_TPB, PT_TPB, 0, st>>>(a, tp)));
  } else {
    SWM_BY_ORDER(order, (div_kernel<ORD, false><<<point_ranges<ORD>(g.n).total / PT_TPB, PT_TPB, 0, st>>>(a, tp)));
  }
  return cudaGetLastError();
}

cudaError_t launch_coriolis(const FieldGeom& g, const double* m64, const double* hu,
                            const double* hv, const double* h, const double* curl, double* cor_u,
                            double* cor_v, cudaStream_t st) {
  coriolis_kernel<<<nblk(6LL * g.n * g.n), TPB, 0, st>>>(g, m64, hu, hv, h, curl, cor_u, cor_v);
  return cudaGetLastError();
}

cudaError_t launch_fill(long long count, double value, double* out, cudaStream_t st) {
  fill_kernel<<<nblk(count), TPB, 0, st>>>(count, value, out);
  return cudaGetLastError();
}

cudaError_t launch_axpby(long long count, double s1, const double* a, double s2, const double* b,
                         double* out, cudaStream_t st) {
  axpby_kernel<<<nblk(count), TPB, 0, st>>>(count, s1, a, s2, b, out);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_sync_vector_t(const FieldGeom& g, const Topology& tp, const double* qw, T* gx,
                                 T* gy, T* edge, cudaStream_t st) {
  const int nb = 6 * (4 * g.n - 4);
  gather_edge_kernel<T><<<nblk(nb), TPB, 0, st>>>(g, gx, EV_GX, gy, EV_GY, edge);
  sync_vector_kernel<T><<<nblk(nb), TPB, 0, st>>>(g, tp, qw, edge, gx, gy);
  return cudaGetLastError();
}
template cudaError_t launch_sync_vector_t<float>(const FieldGeom&, const Topology&, const double*,
                                                 float*, float*, float*, cudaStream_t);
template cudaError_t launch_sync_vector_t<double>(const FieldGeom&, const Topology&, const double*,
                                                  double*, double*, double*, cudaStream_t);

cudaError_t launch_sync_scalar(const FieldGeom& g, const Topology& tp, double* f, double* edge,
                               cudaStream_t st) {
  const int nb = 6 * (4 * g.n - 4);
  gather_edge_kernel<double><<<nblk(nb), TPB, 0, st>>>(g, f, EV_ZETA, nullptr, 0, edge);
  sync_scalar_kernel<double><<<nblk(nb), TPB, 0, st>>>(g, tp, edge, f);
  return cudaGetLastError();
}

cudaError_t launch_sync_vector(const FieldGeom& g, const Topology& tp, const double* qw,
                               double* gx, double* gy, double* edge, cudaStream_t st) {
  return launch_sync_vector_t<double>(g, tp, qw, gx, gy, edge, st);
}

cudaError_t launch_reduce(const FieldGeom& g, int kind, const double* a, const double* b,
                          const double* J, const double* Aw, double hx2, double* partial,
                          int nblocks, double* result, cudaStream_t st) {
  reduce_partial_kernel<<<nblocks, TPB, 0, st>>>(g, kind, a, b, J, Aw, hx2, partial);
  reduce_final_kernel<<<1, TPB, 0, st>>>(partial, nblocks, result);
  return cudaGetLastError();
}

cudaError_t launch_diagnostics(const FieldGeom& g, int order, const Topology& tp, const double* m64,
                               double grav, const double* h, const double* u, const double* v,
                               const double* hs, const double* Aw, double hx2, double* partial,
                               double* result, cudaStream_t st) {
  const OpArgs a{g, u, v, m64, nullptr, 0.0, nullptr, nullptr};
  int blocks = 0;
  SWM_BY_ORDER(order, {
    const int threads = point_ranges<ORD>(g.n).total;
    blocks = threads / PT_TPB < DIAG_BLOCKS ? threads / PT_TPB : DIAG_BLOCKS;
    (diag_kernel<ORD><<<blocks, PT_TPB, 0, st>>>(a, tp, h, hs, Aw, grav, hx2, threads, partial));
  });
  diag_final_kernel<<<1, 32 * DIAG_N, 0, st>>>(partial, blocks, result);
  return cudaGetLastError();
}

cudaError_t launch_axpby_f32pair(long long count, double s1, const float* ahi, const float* alo,
                                 double s2, const float* bhi, const float* blo, float* ohi,
                                 float* olo, cudaStream_t st) {
  const float s1h = (float)s1, s1l = (float)(s1 - (double)s1h);
  const float s2h = (float)s2, s2l = (float)(s2 - (double)s2h);
  axpby_pair_kernel<<<nblk(count), TPB, 0, st>>>(count, s1h, s1l, ahi, alo, s2h, s2l, bhi, blo, ohi,
                                                 olo);
  return cudaGetLastError();
}

cudaError_t launch_fill_f32pair(long long count, double value, float* ohi, float* olo,
                                cudaStream_t st) {
  const float vh = (float)value, vl = (float)(value - (double)vh);
  fill_pair_kernel<<<nblk(count), TPB, 0, st>>>(count, vh, vl, ohi, olo);
  return cudaGetLastError();
}

cudaError_t launch_split_f64(long long count, const double* src, float* hi, float* lo,
                             cudaStream_t st) {
  split_kernel<<<nblk(count), TPB, 0, st>>>(count, src, hi, lo);
  return cudaGetLastError();
}

cudaError_t launch_join_f32pair(long long count, const float* hi, const float* lo, double* dst,
                                cudaStream_t st) {
  join_kernel<<<nblk(count), TPB, 0, st>>>(count, hi, lo, dst);
  return cudaGetLastError();
}

cudaError_t launch_unpack_state(const FieldGeom& g, int nf, const PackedFields& src, void* hi,
                                float* lo, cudaStream_t st) {
  if (nf < 1 || nf > 3 || g.n > 8191) return cudaErrorInvalidValue;
  const unsigned total = (unsigned)(nf * 6LL * g.n * g.n);
  if (lo) unpack_kernel<float><<<nblk(total), TPB, 0, st>>>(g, total, src, (float*)hi, lo);
  else unpack_kernel<double><<<nblk(total), TPB, 0, st>>>(g, total, src, (double*)hi, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_pack_state(const FieldGeom& g, int nf, const void* hi, const float* lo,
                              const PackedFields& dst, cudaStream_t st) {
  if (nf < 1 || nf > 3 || g.n > 8191) return cudaErrorInvalidValue;
  const unsigned total = (unsigned)(nf * 6LL * g.n * g.n);
  if (lo) pack_kernel<float><<<nblk(total), TPB, 0, st>>>(g, total, (const float*)hi, lo, dst);
  else pack_kernel<double><<<nblk(total), TPB, 0, st>>>(g, total, (const double*)hi, nullptr, dst);
  return cudaGetLastError();
}

}  // namespace swm
