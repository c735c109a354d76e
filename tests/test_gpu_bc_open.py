"""The one-launch boundary conditions of a block without wake cut or wall
(bc_open) against the oracle's ordered phases: the smallest block, dimensions
that leave one interior row, rows longer and shorter than a CTA; the state of
every node, the primitives of the viscous kind, and the time step that takes
the boundary nodes' spectral radii from the same launch."""
import numpy as np
import pytest

from cbns3d_cuda_b200 import CBNS_Q, cases
from tests.helpers import rel_linf
from tests.test_gpu_parity import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("viscous", [False, True])
@pytest.mark.parametrize("shape", [(4, 4, 4), (5, 4, 9), (33, 5, 4), (130, 7, 6), (12, 67, 5)])
def test_open_boundaries(shape, viscous):
    c = cases.case_vortex(*shape)
    over = dict(viscous=True, Re=500.0) if viscous else {}
    g, o = pair(c, **over)
    rng = np.random.default_rng(3)
    Q = c.Q0 * (1.0 + 1e-3 * rng.standard_normal(c.Q0.shape))  # every node its own values, ghosts included
    for b in (g, o):
        b.set_conservative(Q)
        if viscous:
            b.calc_primitive(CBNS_Q)
        b.set_bc_calc_primitive(CBNS_Q)
    # the same products, sums and quotients: Q to a rounding, p and T to the
    # rounding of E times E/p ~ 10
    assert rel_linf(g.get_conservative(), o.get_conservative()) <= 1e-15
    if viscous:
        for a, b in zip(g.get_primitive(), o.get_primitive()):
            assert rel_linf(a, b) <= 1e-14
        for b in (g, o):
            b.calc_viscous_terms()
    g.set_time(0.0)
    assert g.run(2) == 2
    rc, t, n = o.solve(2, 1.0e30)
    assert rc == 0 and n == 2
    assert abs(g.get_time()[0] - t) <= 1e-12 * t  # two steps of sums of 1e2 terms
