"""Hyperdiffusion split step on the GPU against the CPU oracle.

The FP64 GPU path follows the oracle's arithmetic (same coefficient tables,
same evaluation order up to the summation of the closure rows), so the bar is
a J-weighted relative L2 difference <= 1e-12 per field for the narrow
Laplacian, the diffusion operator (operator_swm_diff_mod.f90:25-46) and the
drivers' time step of RK4 followed by one explicit Euler diffusion step
(ts2_mod.f90:143-146).  The FP32 context computes the diffusion tendency in
FP32 (within 1e-4 of FP64) and adds it to its compensated state in FP64; its
model steps stay within 1e-5 of the FP64 ones."""
import numpy as np
import pytest

import cubedsphere_sbp_swm_gb300 as swm
from cubedsphere_sbp_swm_gb300 import _abi, initial
import oracle
from gpu_helpers import rel_l2

pytestmark = pytest.mark.gpu

UV = {k: "hordiff_vec_xyz_Ah_sbp_%d_narrow" % k for k in (21, 42, 63)}
H = {k: "hordiff_scalar_Ah_sbp_%d_narrow" % k for k in (21, 42, 63)}


def _state(N, seed=5):
    h, u, v, _ = initial.balanced_zonal(N, 2, 16)
    rng = np.random.default_rng(seed)
    od = oracle.OracleDomain(N, 42)
    h = od.sync_scalar(h + 20.0 * rng.standard_normal(h.shape))
    u, v = od.sync_vector_cov(u + 2.0 * rng.standard_normal(u.shape),
                              v + 2.0 * rng.standard_normal(v.shape))
    return h, u, v


@pytest.mark.parametrize("narrow,N", [(42, 32), (63, 32), (63, 48), (21, 32), (21, 17)])
def test_laplace_matches_oracle(narrow, N):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    od = oracle.OracleDomain(N, 42)
    J = od.geometry()["J"]
    rng = np.random.default_rng(narrow + N)
    f = od.sync_scalar(_state(N)[0] + 5.0 * rng.standard_normal(op.shape))
    fi, fo = op.create_field(), op.create_field()
    fi.upload(f)
    op.laplace(fo, fi, narrow)
    ref = od.laplace(f, narrow)
    assert rel_l2(fo.download(), ref, J) <= 1e-12
    op.laplace(fi, fi, narrow)   # in place
    assert rel_l2(fi.download(), ref, J) <= 1e-12


# The FP64 kernels number the closure columns first: panels of closure columns
# only (6/3 at N=17) and of one and a few inner columns, and of one node more
# than whole warps.
@pytest.mark.parametrize("narrow,N", [(63, 17), (63, 18), (63, 26), (42, 16), (42, 43), (42, 44), (21, 16)])
def test_laplace_small_panels_match_oracle(narrow, N):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    od = oracle.OracleDomain(N, 42)
    f = _state(N)[0]
    fi, fo = op.create_field(), op.create_field()
    fi.upload(f)
    op.laplace(fo, fi, narrow)
    assert rel_l2(fo.download(), od.laplace(f, narrow), od.geometry()["J"]) <= 1e-12


@pytest.mark.parametrize("uv_narrow,h_narrow", [(42, 42), (63, 63), (63, 42), (21, 21), (42, 21)])
def test_diffusion_operator_matches_oracle(uv_narrow, h_narrow):
    N = 32
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    dop = swm.OperatorSWMDiff(op, UV[uv_narrow], 0.03, H[h_narrow], 0.01)
    od = oracle.OracleDomain(N, 42)
    J = od.geometry()["J"]
    h, u, v = _state(N)
    x, t = op.create_stvec(), op.create_stvec()
    x.upload(h, u, v)
    dop.apply(t, x)
    ref = od.diffusion_apply(h, u, v, 0.03, 0.01, uv_narrow, h_narrow)
    for a, b in zip(t.download(), ref):
        assert rel_l2(a, b, J) <= 1e-12


# The FP64 kernels take the fields of a small panel apart, with warps along the
# row on the smallest: panels at either side of the two limits, four fields (three
# and one where the orders differ) and one.
@pytest.mark.parametrize("N,uv_narrow,h_narrow", [(51, 42, 42), (52, 63, 63), (52, 63, 42), (51, 21, 42),
                                                  (160, 42, 42), (161, 42, 63), (161, 21, 21)])
def test_diffusion_operator_at_the_split_limits(N, uv_narrow, h_narrow):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    dop = swm.OperatorSWMDiff(op, UV[uv_narrow], 0.03, H[h_narrow], 0.01)
    od = oracle.OracleDomain(N, 42)
    J = od.geometry()["J"]
    h, u, v = _state(N)
    x, t = op.create_stvec(), op.create_stvec()
    x.upload(h, u, v)
    dop.apply(t, x)
    for a, b in zip(t.download(), od.diffusion_apply(h, u, v, 0.03, 0.01, uv_narrow, h_narrow)):
        assert rel_l2(a, b, J) <= 1e-12


@pytest.mark.parametrize("N,narrow", [(72, 63), (73, 63), (72, 21), (73, 42)])
def test_laplace_at_the_row_warp_limit(N, narrow):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    od = oracle.OracleDomain(N, 42)
    f = _state(N)[0]
    fi, fo = op.create_field(), op.create_field()
    fi.upload(f)
    op.laplace(fo, fi, narrow)
    assert rel_l2(fo.download(), od.laplace(f, narrow), od.geometry()["J"]) <= 1e-12


@pytest.mark.parametrize("order,narrow", [(42, 42), (63, 63), (42, 21)])
def test_model_step_matches_oracle(order, narrow):
    """The 2/1 hyperdiffusion runs after the 4/2 model operator (the Ah
    model operator's orders are 4/2, 4/3 and 6/3)."""
    N, dt, steps = 32, 600.0, 3
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=order, precision="fp64"))
    swm.OperatorSWMDiff(op, UV[narrow], 0.03, H[narrow], 0.01)
    od = oracle.OracleDomain(N, order)
    J = od.geometry()["J"]
    h, u, v = _state(N)
    x = op.create_stvec()
    x.upload(h, u, v)
    op.model_step(x, dt, steps)
    for _ in range(steps):
        h, u, v = od.rk4(h, u, v, dt)
        h, u, v = od.diffusion_step(h, u, v, dt, 0.03, 0.01, narrow, narrow)
    for a, b in zip(x.download(), (h, u, v)):
        assert rel_l2(a, b, J) <= 1e-12


def test_euler_scheme_and_model_step_agree():
    """ExplicitEul1 after RK4 gives the model step's state bit for bit."""
    N, dt = 32, 600.0
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    dop = swm.OperatorSWMDiff(op)
    h, u, v = _state(N)
    a, b = op.create_stvec(), op.create_stvec()
    a.upload(h, u, v)
    b.upload(h, u, v)
    rk4, eul = swm.create_timescheme("rk4"), swm.create_timescheme("explicit_Eul1")
    for _ in range(2):
        rk4.step(a, op, dt)
        eul.step(a, dop, dt)
    op.model_step(b, dt, 2)
    for x, y in zip(a.download(), b.download()):
        assert np.array_equal(x, y)


def test_fp32_model_step_tracks_fp64():
    N, dt, steps = 48, 600.0, 10
    res = {}
    for prec in ("fp64", "fp32"):
        op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision=prec))
        swm.OperatorSWMDiff(op)
        x = op.create_stvec()
        x.upload(*_state(N))
        op.model_step(x, dt, steps)
        res[prec] = x.download()
    J = oracle.OracleDomain(N, 42).geometry()["J"]
    for a, b in zip(res["fp32"], res["fp64"]):
        assert rel_l2(a, b, J) <= 1e-5


@pytest.mark.parametrize("N,narrow", [(16, 42), (20, 42), (17, 63), (23, 63), (40, 63), (16, 21), (40, 21)])
def test_fp32_diffusion_small_panels(N, narrow):
    """The FP32 Laplacian's tiles at the smallest panels the closures allow,
    where a row tile starts inside the closure rows of one end and reaches
    those of the other: the FP32 tendency stays within 1e-4 of FP64."""
    res = {}
    for prec in ("fp64", "fp32"):
        op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision=prec))
        dop = swm.OperatorSWMDiff(op, UV[narrow], 0.03, H[narrow], 0.01)
        x, t = op.create_stvec(), op.create_stvec()
        x.upload(*_state(N))
        dop.apply(t, x)
        res[prec] = t.download()
    J = oracle.OracleDomain(N, 42).geometry()["J"]
    for a, b in zip(res["fp32"], res["fp64"]):
        assert np.all(np.isfinite(a))
        assert rel_l2(a, b, J) <= 1e-4


@pytest.mark.parametrize("N,narrow", [(64, 42), (95, 42), (96, 42), (101, 42), (96, 63), (104, 63), (96, 21), (97, 21)])
def test_fp32_diffusion_tile_ends(N, narrow):
    """The FP32 Laplacian where the last tile but one of a line is moved (panel
    lines of k*32 + 1 nodes and up to the closure rows more), where it just is
    not, and where the move would run into the near closure: the tendency
    stays within 1e-4 of FP64, the small panels' bound."""
    res = {}
    for prec in ("fp64", "fp32"):
        op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision=prec))
        dop = swm.OperatorSWMDiff(op, UV[narrow], 0.03, H[narrow], 0.01)
        x, t = op.create_stvec(), op.create_stvec()
        x.upload(*_state(N))
        dop.apply(t, x)
        res[prec] = t.download()
    J = oracle.OracleDomain(N, 42).geometry()["J"]
    for a, b in zip(res["fp32"], res["fp64"]):
        assert rel_l2(a, b, J) <= 1e-4


@pytest.mark.parametrize("N,narrow", [(64, 42), (96, 42), (101, 42), (97, 63), (104, 63), (96, 21)])
def test_fp32_diffusion_is_the_same_every_time(N, narrow):
    """Nodes in two tiles are written by both, one perhaps by the inner tiles' path:
    in whichever order, the same bits."""
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp32"))
    dop = swm.OperatorSWMDiff(op, UV[narrow], 0.03, H[narrow], 0.01)
    x, t = op.create_stvec(), op.create_stvec()
    x.upload(*_state(N))
    dop.apply(t, x)
    want = t.download()
    for _ in range(20):
        dop.apply(t, x)
        for a, b in zip(t.download(), want):
            assert np.array_equal(a, b)


def test_fp32_diffusion_tendency_tracks_fp64():
    N = 48
    res = {}
    for prec in ("fp64", "fp32"):
        op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision=prec))
        dop = swm.OperatorSWMDiff(op)
        x, t = op.create_stvec(), op.create_stvec()
        x.upload(*_state(N))
        dop.apply(t, x)
        res[prec] = t.download()
    J = oracle.OracleDomain(N, 42).geometry()["J"]
    for a, b in zip(res["fp32"], res["fp64"]):
        assert rel_l2(a, b, J) <= 1e-4


def test_diffusion_conserves_mass_at_scale():
    N = 192
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    dop = swm.OperatorSWMDiff(op)
    x, t = op.create_stvec(), op.create_stvec()
    x.upload(*_state(N))
    dop.apply(t, x)
    th = t.download()[0]
    w = np.zeros(op.shape)
    op._check(op._L.swm_quadrature_weights(op._h, w.ctypes.data_as(_abi._D)))
    assert abs(np.sum(w * th)) <= 1e-11 * np.sum(w * np.abs(th))
    assert np.sum(w * th * x.download()[0]) < 0


def test_errors():
    op = swm.OperatorSWM(swm.ModelConfig(N=32, sbp_order=42, precision="fp64"))
    x, t = op.create_stvec(), op.create_stvec()
    with pytest.raises(swm.SwmError) as e:
        op._check(op._L.swm_apply_diffusion(op._h, t._h, x._h))   # not configured
    assert e.value.code == _abi.SWM_E_INVALID
    with pytest.raises(swm.SwmError) as e:
        swm.OperatorSWMDiff(op, "hordiff_c_biharm_div", 0.03, H[42], 0.01)
    assert e.value.code == _abi.SWM_E_UNSUPPORTED
    with pytest.raises(swm.SwmError) as e:
        swm.create_timescheme("explicit_Eul2")
    assert e.value.code == _abi.SWM_E_UNSUPPORTED
    small = swm.OperatorSWM(swm.ModelConfig(N=16, sbp_order=42, precision="fp64"))
    with pytest.raises(swm.SwmError) as e:   # 17 nodes < 2 x 9 closure rows
        swm.OperatorSWMDiff(small, UV[63], 0.03, H[63], 0.01)
    assert e.value.code == _abi.SWM_E_INVALID
    swm.OperatorSWMDiff(small, UV[42], 0.03, H[42], 0.01)


# ----------------------------------------------------------- laplace_ch_halo4
# hordiff_scalar_Ah / hordiff_vec_xyz_Ah (hordiff_factory_mod.f90:33-40,
# 196-223): the same diffusion pipeline with laplace_ch_halo4 and its ECS_xy
# halo as L; the Ah node mesh is the C-grid oracle's corner mesh.

def test_laplace_ch_on_ah_nodes_matches_oracle():
    N = 32
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    oc = oracle.OracleCDomain(N, 42)
    f = np.random.default_rng(3).standard_normal((6, N + 1, N + 1))
    for order in (2, 4):
        a, b = op.create_field(), op.create_field()
        a.upload(f)
        op.laplace_ch(b, a, order)
        want = oc.laplace_ch(f, order)
        assert np.linalg.norm(b.download() - want) <= 1e-12 * np.linalg.norm(want)
    E = op.ecs_xy_halo(a, 3)
    assert np.abs(E - oc.ecs_xy_halo(f, 3)).max() <= 1e-14 * np.abs(f).max()


def test_hordiff_scalar_ah_tendency_matches_oracle():
    """The h tendency of hordiff_scalar_Ah: -(c^4) L(L(h)), c = coeff a hx,
    L = laplace_ch_halo4 (the oracle's, on the node mesh)."""
    N, coeff = 32, 0.01
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    oc = oracle.OracleCDomain(N, 42)
    dop = swm.OperatorSWMDiff(op, "hordiff_vec_xyz_Ah_sbp_42_narrow", 0.03, "hordiff_scalar_Ah", coeff)
    h, u, v = _state(N)
    vin = op.create_stvec()
    vin.upload(h, u, v)
    vout = vin.create_similar()
    dop.apply(vout, vin)
    c = coeff * 6.371e6 * (0.5 * np.pi / N)
    want = -((c * c) * (c * c)) * oc.laplace_ch(oc.laplace_ch(h, 4), 4)
    got = vout.download()[0]
    assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)


def test_hordiff_vec_xyz_ah_damps_a_solid_rotation_at_the_exact_rate():
    """A solid rotation is an l = 1 field in each Cartesian component, so the
    Cartesian tendency is -4 coeff^4 hx^4 times it; the xyz operator returns
    its projections on b1 and b2 (hordiff_colocated_mod.f90:41-58, kept as
    the reference has it), and the laplace_ch_halo4 pipeline gets there at
    second order four nodes in from the panel edges.  Nearer the edges the
    reference's operator is O(1) off at every resolution: L(L(.)) of its
    Laplacian is about 3% off within two nodes of an edge (the C-grid
    oracle gives the same), and the edge nodes pass contravariant
    projections through the covariant vector sync
    (ecs_Ah_vec_sync_covariant)."""
    errs = []
    for N in (24, 48):
        op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
        dop = swm.OperatorSWMDiff(op, "hordiff_vec_xyz_Ah", 0.03, "hordiff_scalar_Ah", 0.03)
        g = initial.ecs_geometry(N, "ah")
        W = np.cross(np.broadcast_to(np.array([0.0, 0.0, 1.0]), g["r"].shape), g["r"]) * 20.0
        u, v = np.sum(W * g["a1"], -1), np.sum(W * g["a2"], -1)
        h = np.full(u.shape, 5000.0)
        vin = op.create_stvec()
        vin.upload(h, u, v)
        vout = vin.create_similar()
        dop.apply(vout, vin)
        _, tu, tv = vout.download()
        lam = -4.0 * 0.03 ** 4 * (0.5 * np.pi / N) ** 4
        a1, a2 = g["a1"], g["a2"]
        g11, g12, g22 = (a1 * a1).sum(-1), (a1 * a2).sum(-1), (a2 * a2).sum(-1)
        det = g11 * g22 - g12 * g12
        b1 = (g22[..., None] * a1 - g12[..., None] * a2) / det[..., None]
        b2 = (-g12[..., None] * a1 + g11[..., None] * a2) / det[..., None]
        uc, vc = np.sum(W * b1, -1), np.sum(W * b2, -1)
        inner = (slice(None), slice(4, -4), slice(4, -4))
        errs.append(max(np.abs(tu - lam * uc)[inner].max(), np.abs(tv - lam * vc)[inner].max()) /
                    np.abs(lam * uc).max())
    assert errs[0] < 1e-3 and errs[1] < errs[0] / 2.5, errs


def test_laplace_ch_names_need_fp64():
    op = swm.OperatorSWM(swm.ModelConfig(N=24, sbp_order=42, precision="fp32"))
    with pytest.raises(swm.SwmError) as e:
        swm.OperatorSWMDiff(op, "hordiff_vec_xyz_Ah", 0.03, "hordiff_scalar_Ah", 0.01)
    assert e.value.code == _abi.SWM_E_UNSUPPORTED


def test_hordiff_vec_ah_matches_oracle():
    """hordiff_vec_Ah (hordiff_colocated_mod.f90:25-39): each covariant
    component diffused as a scalar, -(c^4) L(L(.)) with laplace_ch_halo4,
    then the covariant vector sync; h by hordiff_scalar_Ah."""
    N, cuv, chh = 32, 0.03, 0.01
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=42, precision="fp64"))
    oc, od = oracle.OracleCDomain(N, 42), oracle.OracleDomain(N, 42)
    dop = swm.OperatorSWMDiff(op, "hordiff_vec_Ah", cuv, "hordiff_scalar_Ah", chh)
    h, u, v = _state(N)
    vin = op.create_stvec()
    vin.upload(h, u, v)
    vout = vin.create_similar()
    dop.apply(vout, vin)
    hx = 0.5 * np.pi / N

    def c4(coeff):
        c = coeff * 6.371e6 * hx
        return -((c * c) * (c * c))

    LL = lambda f: oc.laplace_ch(oc.laplace_ch(f, 4), 4)
    tu, tv = od.sync_vector_cov(c4(cuv) * LL(u), c4(cuv) * LL(v))
    for got, want in zip(vout.download(), (c4(chh) * LL(h), tu, tv)):
        assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
