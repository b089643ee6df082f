"""Set-up data (work units, instance tables, quadrature weights, interpolation
tables) reach the device before the context's stream reads them, also while
the legacy default stream, which that stream does not wait for, is busy.  Each
object is made and used once on an idle GPU and once with work queued there;
one of another shape in between leaves other values in the memory.  Every
table here is below 64 KB, the size up to which a copy on the default stream is
not waited for.

Tolerance: bit-identical results (same calls, same inputs)."""
import numpy as np
import pytest

import cubedsphere_sbp_swm_gb300 as swm
from cubedsphere_sbp_swm_gb300 import initial
from gpu_helpers import busy_default_stream

pytestmark = pytest.mark.gpu


def _start(op, N):
    x = op.create_stvec()
    x.upload(*initial.balanced_zonal(N, 3, 6)[:3])
    return x


def _step(N, order):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=order, precision="fp32"))
    x = _start(op, N)
    swm.RK4().step(x, op, 600.0 * 24 / N, 1)
    out = list(x.download())
    op.set_stage_shape(64, 8)
    swm.RK4().step(x, op, 600.0 * 24 / N, 1)
    return out + list(x.download())


def _diagnostics(N, order):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=order))
    return [np.array(list(op.get_diagnostics(_start(op, N)).values()))]


def _ensemble(N, order):
    sizes = [N, 16]
    ens = swm.Ensemble(swm.ModelConfig(N=N, sbp_order=order, precision="fp32"), sizes, [600.0 * 24 / m for m in sizes])
    for m, size in enumerate(sizes):
        ens.upload(m, *initial.balanced_zonal(size, 3, 6)[:3])
    ens.step(1)
    out = [a for m in range(2) for a in ens.download(m)]
    ens.close()
    return out


def _latlon(N, order):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=order))
    return list(swm.LatLonRegrid(op, 32, 17, "cubic", "covariant").regrid_state(_start(op, N)))


def _laplace_ch(N, order):
    op = swm.OperatorSWM(swm.ModelConfig(N=N, sbp_order=order))
    dop = swm.OperatorSWMDiff(op, "hordiff_vec_xyz_Ah", 0.03, "hordiff_scalar_Ah", 0.01)
    x = _start(op, N)
    y = x.create_similar()
    dop.apply(y, x)
    return list(y.download())


@pytest.mark.parametrize("use", [_step, _diagnostics, _ensemble, _latlon, _laplace_ch])
def test_set_up_while_the_default_stream_is_busy(use):
    want = use(24, 42)
    use(18, 43)
    with busy_default_stream():
        got = use(24, 42)
    assert len(got) == len(want)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
