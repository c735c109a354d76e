"""A batch whose blocks step by themselves between two of its runs.  Such a step
exchanges the roles of the state buffers, so the batch's tables, and the tensor
maps in them, are written anew at the same address before the next run; the
batched stage kernels must then read the new maps."""
from pathlib import Path

import numpy as np
import pytest

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, PREC_FP64, PREC_HYBRID, PREC_SPLIT, Batch, Block, cases, make_params

pytestmark = pytest.mark.gpu

WEIGHTS = Path(cb.__file__).resolve().parent / "data" / "sensor_weights.npz"


def _block(case, precision):
    viscous = bool(case.params.get("viscous"))
    b = Block(make_params(*case.shape, **case.params, precision=precision))
    b.calc_metrics(case.x, case.y, case.z)
    b.set_conservative(case.Q0)
    if viscous:
        b.calc_primitive(CBNS_Q)
    b.set_bc_calc_primitive(CBNS_Q)
    if viscous:
        b.calc_viscous_terms()
    if precision == PREC_HYBRID:
        w = np.load(WEIGHTS)
        b.sensor_load(w["params"], float(w["tau"]))
    b.set_time(0.0)
    return b


def _own_step(b):
    b.set_time(b.step_like_reference(b.get_time()[0], 1.0e30))


@pytest.mark.parametrize("viscous", [False, True])
@pytest.mark.parametrize("precision", [PREC_FP64, PREC_SPLIT, PREC_HYBRID])
def test_blocks_step_between_two_runs(precision, viscous):
    cs, _ = cases.case_batch(4, seed=11, size_lo=(20, 14, 10), size_hi=(44, 30, 18), viscous=viscous)
    for c in cs:
        c.params["bc_mode"] = cb.BC_FARFIELD
    alone, together = ([_block(c, precision) for c in cs] for _ in range(2))
    with Batch(together) as bt:
        for _ in range(3):
            assert bt.run(2) == 2
            for b in together:
                _own_step(b)
        assert bt.run(2) == 2
    for b in alone:
        for _ in range(3):
            assert b.run(2) == 2
            _own_step(b)
        assert b.run(2) == 2
    for a, b in zip(alone, together):
        qa, qb = a.get_conservative(), b.get_conservative()
        # FP64: the same arithmetic; the FP32 fluxes agree to their rounding (a
        # sensor decision at its threshold may differ)
        tol = 1.0e-13 if precision == PREC_FP64 else 1.0e-6
        assert np.max(np.abs(qb - qa)) <= tol * np.max(np.abs(qa))
        assert abs(a.get_time()[0] - b.get_time()[0]) <= tol * a.get_time()[0]
