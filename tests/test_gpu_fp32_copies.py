"""The FP32 copies of the state that the FP32 fluxes, the sensor and the WENO5-face
pass read: whatever wrote the state last wrote them too.

After each kind of writer -- uploads, device initial states, every boundary
mode, stages of a run and of single calls -- the right-hand side of the block is
that of a new block given the downloaded state, bit for bit."""
from pathlib import Path

import numpy as np
import pytest

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, CBNS_QP, Block, cases, make_params

pytestmark = pytest.mark.gpu

WEIGHTS = Path(cb.__file__).resolve().parent / "data" / "sensor_weights.npz"


def _new(c, precision):
    b = Block(make_params(*c.shape, **c.params, precision=precision))
    b.calc_metrics(c.x, c.y, c.z)
    if precision == cb.PREC_HYBRID:
        w = np.load(WEIGHTS)
        b.sensor_load(w["params"], float(w["tau"]))
        b.sensor_audit(97, 1.0e30)  # the audit's sample depends on the step count
    return b


def _case(mode, viscous):
    if mode == "cgrid":  # wake cut and wall
        c = cases.case_naca(48, 24, 6, first=1.0e-3)
        c.params["viscous"] = viscous
    elif mode == "ogrid":
        c = cases.case_naca_ogrid(48, 20, 6, first=2.0e-3, viscous=viscous, start="potential")
    else:
        (c,), _ = cases.case_batch(1, seed=13, size_lo=(37, 22, 13), size_hi=(40, 24, 14), viscous=viscous)
        c.params["bc_mode"] = {"reference": cb.BC_REFERENCE, "farfield": cb.BC_FARFIELD,
                               "characteristic": cb.BC_CHARACTERISTIC}[mode]
    return c


def _check(b, c, precision, which):
    viscous = bool(c.params.get("viscous"))
    if viscous:  # primitives of every node from the state, then the viscous divergence
        b.calc_primitive(which)
        b.calc_viscous_terms()
    got = b.eval_rhs(which)
    with _new(c, precision) as f:
        f.set_conservative(b.get_conservative(which))
        if viscous:
            f.calc_primitive(CBNS_Q)
            f.calc_viscous_terms()
        want = f.eval_rhs(CBNS_Q)
    assert np.isfinite(want).all() and np.array_equal(got, want)


@pytest.mark.parametrize("precision", [cb.PREC_SPLIT, cb.PREC_HYBRID])
@pytest.mark.parametrize("viscous", [False, True])
@pytest.mark.parametrize("mode", ["reference", "farfield", "characteristic", "cgrid", "ogrid"])
def test_every_writer_writes_the_copy(mode, viscous, precision):
    c = _case(mode, viscous)
    with _new(c, precision) as b:
        if c.Q0 is None:
            b.initial_condition()
            b.calc_conservative(CBNS_Q)
        else:
            b.set_conservative(c.Q0)
        _check(b, c, precision, CBNS_Q)
        if viscous:
            b.calc_primitive(CBNS_Q)
        b.set_bc_calc_primitive(CBNS_Q)
        _check(b, c, precision, CBNS_Q)
        b.set_time(0.0)
        assert b.run(2) == 2
        _check(b, c, precision, CBNS_Q)
        if viscous:
            b.calc_primitive(CBNS_Q)
            b.set_bc_calc_primitive(CBNS_Q)
            b.calc_viscous_terms()
        dt = b.calc_dt()
        for stage in (1, 2, 3):
            which = CBNS_QP if stage < 3 else CBNS_Q
            b.calc_numerical_flux(CBNS_Q if stage == 1 else CBNS_QP)
            b.update_rk3(dt, stage)
            b.set_bc_calc_primitive(which)
            _check(b, c, precision, which)


@pytest.mark.parametrize("precision", [cb.PREC_SPLIT, cb.PREC_HYBRID])
def test_device_initial_state(precision):
    x, y, z = cases.stretched_skewed_box(30, 22, 14)
    c = cases.Case("blast", x, y, z, dict(Mach=2.6, gamma=1.4, i_begin=1, i_end=0), None, t_end=1.0, nsteps=1)
    with _new(c, precision) as b:
        b.init_case(1, x, y, z, [0.1, 8.0, 0.2])
        _check(b, c, precision, CBNS_Q)
