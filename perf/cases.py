"""Performance cases: the work that users of this framework have it do.

Every case goes through the public Python objects (OperatorSWM, StvecSWM, RK4,
Ensemble, trajectory, ...).  The kinds are

  run       a stretch of the model: an initial state, `steps` time steps (RK4,
            or RK4 + hyperdiffusion with "diffusion"), the fields copied to
            page-locked host arrays, on the Ah or the C grid, FP64 or FP32;
  ensemble  members of several resolutions uploaded, advanced together and
            read back;
  gradient  a differentiated forecast: the trajectory forward, a quadratic
            misfit of the final depth and its gradient with respect to x0;
  exchange  a host model that hands its state over for every step: upload,
            one step, download, two states taking turns;
  analysis  an output step: the global diagnostics, the depth gradient, the
            vorticity and the divergence, and the state on a lat-lon grid.

exact() restates the Ah model (operators, cube-edge averages, RK4) in plain
FP64 torch; its gradient is torch's own.  The C grid, the narrow-stencil
hyperdiffusion and the lat-lon interpolation have long coefficient tables of
their own and are held to the bounds of their types alone.
"""
import math

import numpy as np
import torch

import cubedsphere_sbp_swm_gb300 as swm
from cubedsphere_sbp_swm_gb300 import adjoint

RADIUS, GRAV, OMEGA = 6.371e6, 9.80616, 7.292e-5
DEPTH = 5960.0
MEMBER_N = (48, 96, 192)  # member resolutions of an ensemble


def listed():
    return [
        # the smallest useful panels: short climate-style integrations, where
        # launches and latency are all there is
        dict(name="run_ah_fp32_n48_d42", kind="run", grid="Ah", N=48, order=42, precision="fp32",
             diffusion=False, steps=40),
        # the headline step of the benchmark, FP32 form and FP64 form
        dict(name="run_ah_fp32_n384_d42", kind="run", grid="Ah", N=384, order=42, precision="fp32",
             diffusion=False, steps=20),
        dict(name="run_ah_fp64_n384_d42", kind="run", grid="Ah", N=384, order=42, precision="fp64",
             diffusion=False, steps=10),
        # the large instance of the benchmark
        dict(name="run_ah_fp32_n1024_d63", kind="run", grid="Ah", N=1024, order=63, precision="fp32",
             diffusion=False, steps=20),
        # the drivers' time step with hyperdiffusion: production runs
        dict(name="model_ah_fp32_n384_d42", kind="run", grid="Ah", N=384, order=42, precision="fp32",
             diffusion=True, steps=10),
        dict(name="model_ah_fp64_n201_d63", kind="run", grid="Ah", N=201, order=63, precision="fp64",
             diffusion=True, steps=6),
        # the C-grid family: RK4 in FP64, the namelist's model step in FP32
        dict(name="run_c_fp64_n384_42", kind="run", grid="C", N=384, order=42, precision="fp64",
             diffusion=False, steps=8),
        dict(name="model_c_fp32_n384_42", kind="run", grid="C", N=384, order=42, precision="fp32",
             diffusion=True, steps=10),
        # forecasts with perturbed members
        dict(name="ensemble_fp32_9", kind="ensemble", members=9, order=42, precision="fp32", steps=120),
        # variational assimilation: forward and backward through the model
        dict(name="gradient_fp64_n192_d42", kind="gradient", N=192, order=42, precision="fp64", steps=24,
             snapshots=6),
        # coupling to a host model every step
        dict(name="exchange_fp32_n384_d42", kind="exchange", N=384, order=42, precision="fp32"),
        # an output step
        dict(name="analysis_fp64_n130_d42", kind="analysis", N=130, order=42, precision="fp64"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["run"] * 6 + ["ensemble", "gradient", "exchange", "analysis"])
    precision = rng.choice(["fp32", "fp64"])
    top = 1024 if precision == "fp32" else 384
    order = rng.choice([42, 43, 63])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 12), order=order, precision=precision,
                    steps=rng.randint(20, 90) if precision == "fp32" else rng.randint(4, 20))
    if kind == "gradient":
        steps = rng.randint(4, 24)
        return dict(kind=kind, N=_log_uniform(rng, 32, 192), order=order, precision=precision, steps=steps,
                    snapshots=rng.randint(2, min(steps, 8)))
    if kind == "exchange":
        return dict(kind=kind, N=_log_uniform(rng, 24, 640), order=order, precision=precision)
    if kind == "analysis":
        return dict(kind=kind, N=_log_uniform(rng, 24, 256), order=order, precision="fp64")
    grid = rng.choice(["Ah", "C"])
    if grid == "C":
        order, top = rng.choice([21, 42]), 384
    N = _log_uniform(rng, 16, top)
    steps = rng.randint(4, 20)
    if N > 256 and precision == "fp64":
        steps = min(steps, 6)
    return dict(kind=kind, grid=grid, N=N, order=order, precision=precision, diffusion=rng.random() < 0.4,
                steps=steps)


# --------------------------------------------------------------- the inputs
_EX = ((-1, 0, 0), (0, 0, -1), (1, 0, 0), (0, 0, 1), (1, 0, 0), (1, 0, 0))
_EY = ((0, 1, 0), (0, 1, 0), (0, 1, 0), (0, 1, 0), (0, 0, 1), (0, 0, -1))
_EN = ((0, 0, 1), (-1, 0, 0), (0, 0, -1), (1, 0, 0), (0, 1, 0), (0, -1, 0))


def _faces(v):
    """A prototype-face vector field (ny, nx, 3) on the six panels."""
    return np.stack([v @ np.array([_EX[p], _EY[p], [-c for c in _EN[p]]], float) for p in range(6)])


def _geometry(N, half_i=False, half_j=False):
    """Points r and covariant basis a1, a2 of the unit equiangular cubed
    sphere, (6, ny, nx, 3), on the nodes or shifted half a cell."""
    hx = 0.5 * math.pi / N
    al = -0.25 * math.pi + hx * (np.arange(N if half_i else N + 1) + (0.5 if half_i else 0.0))
    be = -0.25 * math.pi + hx * (np.arange(N if half_j else N + 1) + (0.5 if half_j else 0.0))
    X, Y = np.broadcast_arrays(np.tan(al)[None, :], np.tan(be)[:, None])
    s = np.sqrt(1.0 + X * X + Y * Y)
    r = np.stack([X, Y, np.ones_like(X)], -1) / s[..., None]
    a1 = ((1 + X * X) / s**3)[..., None] * np.stack([1 + Y * Y, -X * Y, -X], -1)
    a2 = ((1 + Y * Y) / s**3)[..., None] * np.stack([-X * Y, 1 + X * X, -Y], -1)
    return _faces(r), _faces(a1), _faces(a2)


def _initial(N, seed, grid="Ah"):
    """A balanced zonal flow with a 10 m perturbation of the depth and a 1 m/s
    one of the wind: (h, u, v), u and v covariant, each on its own mesh."""
    rng = np.random.RandomState(seed % (1 << 31))
    u0 = rng.uniform(20.0, 40.0)
    wave = rng.uniform(-8.0, 8.0, (8, 3))
    phase = rng.uniform(0.0, 2.0 * math.pi, 8)
    amp = rng.uniform(2.0, 5.0, 8)
    gust = rng.uniform(-0.5, 0.5, (8, 3))
    meshes = [(False, False)] * 3 if grid == "Ah" else [(True, True), (False, True), (True, False)]
    out = []
    for c, (hi, hj) in enumerate(meshes):
        if c == 0 or grid == "C":
            r, a1, a2 = _geometry(N, hi, hj)
        if c == 0:
            f = DEPTH - (RADIUS * OMEGA * u0 + 0.5 * u0 * u0) / GRAV * (r[..., 2] ** 2 - 1.0 / 3.0)
            for k in range(8):
                f = f + amp[k] * np.sin(r @ wave[k] + phase[k])
        else:
            a = a1 if c == 1 else a2
            f = u0 * (r[..., 0] * a[..., 1] - r[..., 1] * a[..., 0])
            for k in range(8):
                f = f + (a @ gust[k]) * np.sin(r @ wave[k] - phase[k])
        out.append(np.ascontiguousarray(f))
    return out


def _time_step(case, N):
    """Stable steps: Courant number about 0.55 on the Ah grid, 0.4 on the C grid."""
    return (37.5 if case.get("grid") == "C" else 60.0) * 384.0 / N


def _pinned(shapes):
    tensors = [torch.empty(sh, dtype=torch.float64, pin_memory=True) for sh in shapes]
    return tensors, tuple(t.numpy() for t in tensors)


def _member_N(case):
    return [MEMBER_N[m % len(MEMBER_N)] for m in range(case["members"])]


def _observed(N, seed):
    """Observed depths of the misfit."""
    return _initial(N, seed + 7919)[0]


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, rk4=swm.create_timescheme("rk4"))
    if kind == "ensemble":
        Ns = _member_N(case)
        base = swm.ModelConfig(N=Ns[0], sbp_order=case["order"], precision=case["precision"])
        st["ens"] = swm.Ensemble(base, Ns, [_time_step(case, N) for N in Ns])
        st["x0"] = []
        for m, N in enumerate(Ns):
            _, x = _pinned([(6, N + 1, N + 1)] * 3)
            for a, b in zip(x, _initial(N, seed * 64 + m)):
                a[...] = b
            st["x0"].append(x)
        return st
    N = case["N"]
    grid = case.get("grid", "Ah")
    names = swm.c_grid_names(case["order"]) if grid == "C" else None
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=case["order"], precision=case["precision"], names=names))
    st["op"], st["dt"] = op, _time_step(case, N)
    x0 = _initial(N, seed, grid)
    if kind == "run":
        st["x0"], st["x"] = op.create_stvec(), op.create_stvec()
        st["x0"].upload(*x0)
        if case["diffusion"]:
            if grid == "C":
                st["diff"] = swm.OperatorSWMDiff(op)
            else:
                nn = 63 if case["order"] == 63 else 42
                st["diff"] = swm.OperatorSWMDiff(op, f"hordiff_vec_xyz_Ah_sbp_{nn}_narrow", 0.03,
                                                 f"hordiff_scalar_Ah_sbp_{nn}_narrow", 0.01)
        st["out"], st["host"] = _pinned(op.state_shapes)
    elif kind == "gradient":
        st["x0"] = torch.as_tensor(np.stack(x0), device="cuda")
        st["obs"] = torch.as_tensor(_observed(N, seed), device="cuda")
        st["weights"] = torch.as_tensor(adjoint.quadrature_weights(op), device="cuda")
        st["runner"] = adjoint.CheckpointedRK4(op, st["dt"], case["steps"], case["snapshots"])
    elif kind == "exchange":
        st["turn"] = 0
        st["slots"] = []
        for _ in range(2):
            _, src = _pinned(op.state_shapes)
            for a, b in zip(src, x0):
                a[...] = b
            out, dst = _pinned(op.state_shapes)
            st["slots"].append((op.create_stvec(), src, dst, out))
    else:
        st["x"] = op.create_stvec()
        st["x"].upload(*x0)
        st["f"] = {k: op.create_field() for k in ("h", "u", "v", "ut", "vt", "gx", "gy", "curl", "div")}
        for k, a in zip("huv", x0):
            st["f"][k].upload(a)
        st["latlon"] = swm.LatLonRegrid(op, 4 * N, 2 * N + 1, "cubic", "covariant")
    return st


# ---------------------------------------------------------------------- run
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "run":
        st["x"].assign_s1v1(1.0, st["x0"])
        if case["diffusion"]:
            st["op"].model_step(st["x"], st["dt"], case["steps"])
        else:
            st["rk4"].step(st["x"], st["op"], st["dt"], case["steps"])
        st["x"].download_async(st["host"])
        return st["out"]
    if kind == "ensemble":
        ens = st["ens"]
        for m, x in enumerate(st["x0"]):
            ens.upload(m, *x)
        ens.step(case["steps"])
        return [ens.download(m) for m in range(len(ens))]
    if kind == "gradient":
        x0 = st["x0"].detach().requires_grad_(True)
        xT = adjoint.trajectory(x0, st["runner"])
        misfit = 0.5 * (st["weights"] * (xT[0] - st["obs"]) ** 2).sum()
        (grad,) = torch.autograd.grad(misfit, x0)
        return [xT.detach(), grad]
    if kind == "exchange":
        x, src, dst, out = st["slots"][st["turn"]]
        st["turn"] ^= 1
        x.upload_async(*src)
        st["rk4"].step(x, st["op"], st["dt"])
        x.download_async(dst)
        return out
    op, f = st["op"], st["f"]
    diag = op.get_diagnostics(st["x"])
    op.calc_grad(f["gx"], f["gy"], f["h"])
    op.calc_curl(f["curl"], f["u"], f["v"])
    op.co2contra(f["ut"], f["vt"], f["u"], f["v"])
    op.calc_div(f["div"], f["ut"], f["vt"])
    fields = [f[k].download() for k in ("gx", "gy", "curl", "div")]
    return dict(diag=np.array([diag[k] for k in swm.DIAG_KEYS]), fields=fields,
                latlon=list(st["latlon"].regrid_state(st["x"])))


# --------------------------------------------------------------------- work
# One RK4 stage is a pass over the grid: the stage input (3 values a point),
# the metric (5 on the Ah grid, 8 on the C grid's meshes) and the RK sums are
# read, the next stage input and sum are written: 68 (FP64) or 77 (FP32, whose
# state is a pair) values a point and step on the Ah grid.
def _step_work(N, grid, order, precision, diffusion):
    points = 6.0 * (N + 1) ** 2
    size = 4 if precision == "fp32" else 8
    words = (77 if precision == "fp32" else 68) + (12 if grid == "C" else 0)
    flops = 4 * (190 if grid == "C" else {42: 100, 43: 100, 63: 125}.get(order, 100))
    if diffusion:
        # state in and out, one intermediate of 4 fields out and in, the metric
        # and basis vectors twice
        words += (12 if precision == "fp32" else 6) + 8 + 2 * 10
        flops += 600 if grid == "Ah" else 250
    return points * words * size, points * flops


def work(case):
    kind = case["kind"]
    grid = case.get("grid", "Ah")
    if kind == "ensemble":
        per = [_step_work(N, "Ah", case["order"], case["precision"], False) for N in _member_N(case)]
        state = sum(2 * 3 * 8 * 6 * (N + 1) ** 2 for N in _member_N(case))
        return {"bytes": case["steps"] * sum(b for b, _ in per) + state,
                "flops": case["steps"] * sum(f for _, f in per)}
    N = case["N"]
    points = 6 * (N + 1) ** 2
    b, f = _step_work(N, grid, case["order"], case["precision"], case.get("diffusion", False))
    if kind == "run":
        return {"bytes": case["steps"] * b + 24 * points, "flops": case["steps"] * f}
    if kind == "gradient":
        # forward once; backward: the stage states again and the transposed stages
        return {"bytes": 3 * case["steps"] * b + 4 * 24 * points, "flops": 3 * case["steps"] * f}
    if kind == "exchange":
        return {"bytes": b + 48 * points, "flops": f}
    # state, fields and metric read, four fields and three lat-lon planes written
    return {"bytes": 8 * (points * (3 + 3 + 5 + 2 + 4) + 3 * 4 * N * (2 * N + 1)), "flops": 150.0 * points}


# -------------------------------------------------------------------- exact
# SBP first derivatives: closure rows at the left end (the right end mirrors
# them with the opposite sign), interior stencil, norm at the edge.
def _tables(order):
    if order == 42:
        rows = [[-24 / 17, 59 / 34, -4 / 17, -3 / 34], [-1 / 2, 0, 1 / 2],
                [4 / 43, -59 / 86, 0, 59 / 86, -4 / 43], [3 / 98, 0, -59 / 98, 0, 32 / 49, -4 / 49]]
    elif order == 43:
        rows = [[-1.8280236842718398, 2.978054584697369, -1.4653148294044123, 0.3078538227474199,
                 0.008136925288119662, -0.0007068190566565205],
                [-0.37814159126691327, -0.31480210500706657, 0.707290999364066, 0.04835554461933453,
                 -0.06866771096803422, 0.005964863258613564],
                [0.1162478575921292, -0.8028500807354999, 0.21558841368737428, 0.5078566674295846,
                 -0.03231754093993847, -0.004525317033649745],
                [-0.010287398573128293, 0.12592344801071614, -0.7341531396449149, 0.04979271660173103,
                 0.6506171865540596, -0.08189281294846368]]
    else:
        a = [13649 / 43200, 12013 / 8640, 2711 / 4320, 5359 / 4320, 7877 / 8640, 43801 / 43200]
        q = 5591070156686698065364559 / 7931626489314500743872000
        Q = np.zeros((6, 9))
        Q[0, :6] = [-1 / 2, -953 / 16200 + q, 715489 / 259200 - 4 * q, -62639 / 14400 + 6 * q,
                    147127 / 51840 - 4 * q, -89387 / 129600 + q]
        Q[1, 2:6] = [-57139 / 8640 + 10 * q, 745733 / 51840 - 20 * q, -18343 / 1728 + 15 * q,
                     240569 / 86400 - 4 * q]
        Q[2, 3:6] = [-176839 / 12960 + 20 * q, 242111 / 17280 - 20 * q, -182261 / 43200 + 6 * q]
        Q[3, 4:7] = [-165041 / 25920 + 10 * q, 710473 / 259200 - 4 * q, 1 / 60]
        Q[4, 5:8] = [q, -3 / 20, 1 / 60]
        Q[5, 6:9] = [3 / 4, -3 / 20, 1 / 60]
        Q[:, :6] -= np.triu(Q[:, :6], 1).T  # the off-diagonal part is antisymmetric
        rows = [list(Q[k] / a[k]) for k in range(6)]
        return rows, [-1 / 60, 3 / 20, -3 / 4, 0, 3 / 4, -3 / 20, 1 / 60], a
    return rows, [1 / 12, -2 / 3, 0, 2 / 3, -1 / 12], [17 / 48, 59 / 48, 43 / 48, 49 / 48]


class _Exact:
    """The Ah model in FP64 torch, fields of shape (6, n, n)."""

    def __init__(self, N, order):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.N, self.n, n = N, N + 1, N + 1
        rows, mid, edge = _tables(order)
        D = np.zeros((n, n))
        half = len(mid) // 2
        for k in range(n):
            if k < len(rows):
                D[k, :len(rows[k])] = rows[k]
            elif k >= n - len(rows):
                row = rows[n - 1 - k]
                D[k, n - len(row):] = [-x for x in reversed(row)]
            else:
                D[k, k - half:k + half + 1] = mid
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)  # noqa: E731
        self.D = t(D)
        self.hx = 0.5 * math.pi / N
        r, a1, a2 = _geometry(N)
        tan = np.tan(-0.25 * math.pi + self.hx * np.arange(n))
        X, Y = np.broadcast_arrays(tan[None, :], tan[:, None])
        s2 = 1.0 + X * X + Y * Y
        A, B = 1.0 + X * X, 1.0 + Y * Y
        self.J, self.q1, self.q2, self.q3 = t(A * B / s2**1.5), t(s2 / A), t(s2 * X * Y / (A * B)), t(s2 / B)
        self.f = t(2.0 * OMEGA * r[..., 2])
        w = np.ones(n)
        w[:len(edge)] = edge
        w[n - len(edge):] = edge[::-1]
        self.w = self.J * t(self.hx**2 * w[None, :] * w[:, None])
        # copies of a panel-edge node: its point on the cube, in whole numbers
        k = 2 * np.arange(n) - N
        kx, ky = np.broadcast_arrays(k[None, :], k[:, None])
        cube = np.rint(_faces(np.stack([kx, ky, np.full_like(kx, N)], -1).astype(float))).astype(np.int64)
        at = np.nonzero(((np.abs(cube) == N).sum(-1) > 1).reshape(-1))[0]
        _, group, count = np.unique(cube.reshape(-1, 3)[at], axis=0, return_inverse=True, return_counts=True)
        self.at, self.group = torch.as_tensor(at, device=dev), torch.as_tensor(group.reshape(-1), device=dev)
        self.count = t(count)
        pick = lambda v: t(v.reshape(-1, 3)[at])  # noqa: E731
        self.a1, self.a2 = pick(a1), pick(a2)
        m = lambda v: v.expand(6, n, n).reshape(-1)[self.at][:, None]  # noqa: E731
        self.b1 = m(self.q1) * self.a1 + m(self.q2) * self.a2
        self.b2 = m(self.q2) * self.a1 + m(self.q3) * self.a2
        self.to = t

    def dx(self, f):
        return f @ self.D.T / (self.hx * RADIUS)

    def dy(self, f):
        return self.D @ f / (self.hx * RADIUS)

    def _mean(self, v):
        s = torch.zeros((len(self.count),) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, self.group, v)
        return (s / (self.count[:, None] if v.dim() > 1 else self.count))[self.group]

    def sync(self, f):
        flat = f.reshape(-1)
        return flat.index_copy(0, self.at, self._mean(flat[self.at])).reshape(f.shape)

    def grad(self, f):
        gx, gy = self.dx(f).reshape(-1), self.dy(f).reshape(-1)
        g = self._mean(gx[self.at][:, None] * self.b1 + gy[self.at][:, None] * self.b2)
        return (gx.index_copy(0, self.at, (g * self.a1).sum(-1)).reshape(f.shape),
                gy.index_copy(0, self.at, (g * self.a2).sum(-1)).reshape(f.shape))

    def contra(self, u, v):
        return self.q1 * u + self.q2 * v, self.q2 * u + self.q3 * v

    def curl(self, u, v):
        return self.sync((self.dx(v) - self.dy(u)) / self.J)

    def div(self, ut, vt):
        return self.sync((self.dx(self.J * ut) + self.dy(self.J * vt)) / self.J)

    def tendency(self, x):
        h, u, v = x
        ut, vt = self.contra(u, v)
        gx, gy = self.grad(0.5 * (u * ut + v * vt) + GRAV * h)
        fz = self.f + self.curl(u, v)
        return torch.stack([-self.div(h * ut, h * vt), -gx + fz * self.J * vt, -gy - fz * self.J * ut])

    def steps(self, x, dt, count):
        for _ in range(count):
            k1 = self.tendency(x)
            k2 = self.tendency(x + 0.5 * dt * k1)
            k3 = self.tendency(x + 0.5 * dt * k2)
            k4 = self.tendency(x + dt * k3)
            x = x + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for m, N in enumerate(_member_N(case)):
            M = _Exact(N, case["order"])
            out.append(list(M.steps(M.to(np.stack(_initial(N, seed * 64 + m))), _time_step(case, N), case["steps"])))
        return out
    if case.get("grid") == "C" or case.get("diffusion"):
        return None
    N = case["N"]
    M = _Exact(N, case["order"])
    dt = _time_step(case, N)
    x0 = M.to(np.stack(_initial(N, seed)))
    if kind in ("run", "exchange"):
        return list(M.steps(x0, dt, case.get("steps", 1)))
    if kind == "gradient":
        x0.requires_grad_(True)
        xT = M.steps(x0, dt, case["steps"])
        (grad,) = torch.autograd.grad(0.5 * (M.w * (xT[0] - M.to(_observed(N, seed))) ** 2).sum(), x0)
        return [xT.detach(), grad]
    h, u, v = x0
    ut, vt = M.contra(u, v)
    gx, gy = M.grad(h)
    curl, div = M.curl(u, v), M.div(ut, vt)
    ke = float((0.5 * h * (ut * u + vt * v) * M.w).sum())
    pe = float((0.5 * GRAV * h * h * M.w).sum())
    diag = [float(h.min()), float(h.max()), float((h * M.w).sum()), ke + pe, ke, pe,
            float((0.5 * (curl + M.f) ** 2 / h * M.w).sum())]
    return dict(diag=np.array(diag), fields=[gx, gy, curl, div], latlon=[None, None, None])
