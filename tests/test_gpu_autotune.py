"""cbns_autotune times stages on the block itself: the state, the time and a
finished run's mark stand afterwards, and the steps that follow are those of a
block set by hand to the pair it chose."""
import numpy as np
import pytest

from cbns3d_cuda_b200 import CBNS_Q, PREC_FP64, PREC_SPLIT, Block, cases, make_params

pytestmark = pytest.mark.gpu


def _block(c, precision):
    b = Block(make_params(*c.shape, **c.params, precision=precision))
    b.calc_metrics(c.x, c.y, c.z)
    b.set_conservative(c.Q0)
    b.set_bc_calc_primitive(CBNS_Q)
    b.set_time(0.0)
    return b


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_SPLIT])
@pytest.mark.parametrize("shape", [(20, 14, 10), (67, 34, 21)])
def test_autotune_leaves_the_block_as_it_was(shape, precision):
    c = cases.case_blast(*shape)
    a, b = _block(c, precision), _block(c, precision)
    assert a.run(4) == 4 and b.run(4) == 4
    t = a.get_time()[0]
    assert a.run(5, t) == 0 and b.run(5, t) == 0  # at its end time: the run is finished
    q = a.get_conservative().copy()
    v = a.autotune()
    assert np.array_equal(a.get_conservative(), q) and a.get_time()[0] == t
    b.stage_variant(v)
    b.stage_kchunk(a.stage_kchunk())
    assert a.run(3) == 3 and b.run(3) == 3
    assert np.array_equal(a.get_conservative(), b.get_conservative()) and a.get_time() == b.get_time()
