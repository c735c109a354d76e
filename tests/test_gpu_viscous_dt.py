"""The time step of a viscous run, whose spectral radii the node kernel forms in
FP64 only where FP32 bounds let them be the largest, against the sweep over
every node.  Flows where the convective part is all but everything and flows
where the viscous part is; both forms of the viscous part."""
import numpy as np
import pytest

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, Block, cases, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [cb.PREC_FP64, cb.PREC_SPLIT])
@pytest.mark.parametrize("form", [cb.DTV_REFERENCE, cb.DTV_FULL])
@pytest.mark.parametrize("Re", [1.0, 50.0, 1.0e5])
def test_time_step_is_the_largest_spectral_radius(precision, form, Re):
    blocks, _ = cases.case_batch(3, seed=21, size_lo=(12, 10, 6), size_hi=(70, 40, 24), viscous=True)
    for c in blocks:
        c.params.update(bc_mode=cb.BC_FARFIELD, Re=Re)
        with Block(make_params(*c.shape, **c.params, precision=precision, dt_viscous=form)) as b:
            b.calc_metrics(c.x, c.y, c.z)
            b.set_conservative(c.Q0)
            b.calc_primitive(CBNS_Q)
            b.set_bc_calc_primitive(CBNS_Q)
            b.calc_viscous_terms()
            b.set_time(0.0)
            for _ in range(3):
                assert b.run(1) == 1
                dt = b.calc_dt()  # from the step's own kernels
                b.calc_metrics(c.x, c.y, c.z)  # the spectral radii are formed anew
                full = b.calc_dt()
                # the same formulas, contracted differently: 20 roundings; split: mu, kept in FP32 (4 of 2^-24)
                tol = 20 * 2.0 ** -53 if precision == cb.PREC_FP64 else 4 * 2.0 ** -24
                assert abs(dt - full) <= tol * full
