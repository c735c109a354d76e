"""A node that stage 3 leaves with a pressure slightly below zero makes the time
step a NaN, whichever nodes were met before it.

The node's pressure is within the rounding that the FP32 bound of the spectral
radius adds to it (1e-6 of its energy), so the bound alone is positive and far
below the other nodes' values.  The state comes through stage 3 unchanged: it
is uniform but for that node, and the step has length zero.
"""
from pathlib import Path

import numpy as np
import pytest

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, CBNS_QP, Block, make_params

pytestmark = pytest.mark.gpu

WEIGHTS = Path(cb.__file__).resolve().parent / "data" / "sensor_weights.npz"
N = 12


def _block(precision):
    b = Block(make_params(N, N, N, Mach=100.0, bc_mode=cb.BC_FARFIELD, precision=precision))
    k, j, i = np.meshgrid(*(np.linspace(0.0, 1.0, N),) * 3, indexing="ij")
    b.calc_metrics(i, j, k)
    if precision == cb.PREC_HYBRID:
        w = np.load(WEIGHTS)
        b.sensor_load(w["params"], float(w["tau"]))
        b.sensor_audit(97, 1.0e30)
    b.stage_kchunk(N - 2)  # one CTA: the other planes come before the node's
    return b


@pytest.mark.parametrize("precision", [cb.PREC_FP64, cb.PREC_SPLIT, cb.PREC_HYBRID])
@pytest.mark.parametrize("p_node, nan", [(0.02, False), (1.0e-7, False), (-2.0e-5, True), (-7.0e-5, True)])
def test_negative_pressure_of_stage_3_ends_the_steps(precision, p_node, nan):
    p = np.full((N + 4,) * 3, 0.02)
    p[N, 6, 6] = p_node  # interior node (4, 4, N-2): the last plane
    Q = np.zeros(p.shape + (5,))
    Q[..., 0], Q[..., 1] = 1.0, 20.0
    Q[..., 4] = p / 0.4 + 200.0
    with _block(precision) as b:
        b.set_conservative(Q)
        b.set_bc_calc_primitive(CBNS_Q)
        for stage, src in ((1, CBNS_Q), (2, CBNS_QP), (3, CBNS_QP)):
            b.calc_numerical_flux(src)
            b.update_rk3(0.0, stage)
            b.set_bc_calc_primitive(CBNS_QP if stage < 3 else CBNS_Q)
        out = b.get_conservative(CBNS_Q).reshape(Q.shape)
        assert np.isfinite(out).all() and np.abs(out - Q).max() < 1.0e-12
        if nan:
            with pytest.raises(cb.CbnsError):
                b.calc_dt()
        else:
            assert np.isfinite(b.calc_dt())
