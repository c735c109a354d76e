"""cbns_autotune on a hybrid block, whose kernels it times on the sensor's
decisions for the state: state, time and a finished run's mark stand afterwards,
and the steps that follow are those of a block set by hand to its choice."""
from pathlib import Path

import numpy as np
import pytest

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import CBNS_Q, Block, cases, make_params

pytestmark = pytest.mark.gpu

WEIGHTS = Path(cb.__file__).resolve().parent / "data" / "sensor_weights.npz"


@pytest.mark.parametrize("shape", [(20, 14, 10), (67, 34, 21)])
def test_autotune_leaves_a_hybrid_block_as_it_was(shape):
    c = cases.case_blast(*shape)
    w = np.load(WEIGHTS)
    pair = []
    for _ in range(2):
        b = Block(make_params(*c.shape, **c.params, precision=cb.PREC_HYBRID))
        b.calc_metrics(c.x, c.y, c.z)
        b.sensor_load(w["params"], float(w["tau"]))
        b.set_conservative(c.Q0)
        b.set_bc_calc_primitive(CBNS_Q)
        b.set_time(0.0)
        pair.append(b)
    a, b = pair
    assert a.run(4) == 4 and b.run(4) == 4
    t = a.get_time()[0]
    assert a.run(5, t) == 0 and b.run(5, t) == 0  # at its end time: the run is finished
    q = a.get_conservative().copy()
    v = a.autotune()
    assert np.array_equal(a.get_conservative(), q) and a.get_time()[0] == t
    b.stage_variant(v)
    b.stage_kchunk(a.stage_kchunk())
    assert a.run(4) == 4 and b.run(4) == 4
    assert np.array_equal(a.sensor_mask()[0], b.sensor_mask()[0])
    assert np.array_equal(a.get_conservative(), b.get_conservative()) and a.get_time() == b.get_time()
