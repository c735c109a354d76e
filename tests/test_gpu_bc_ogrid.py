"""The one-launch O-grid boundary conditions (bc_ogrid) against the oracle's
ordered passes at the edges of its range: the shortest periodic line the wrap
allows (every stored point copied to both sides), four points along the span,
and a wall-normal line of four; Q of every node, the primitives of the viscous
kind, every copy across the seam bit for bit."""
import numpy as np
import pytest

from cbns3d_cuda_b200 import CBNS_Q, OGRID_WRAP, cases
from tests.helpers import rel_linf
from tests.test_gpu_parity import pair

pytestmark = pytest.mark.gpu
W = OGRID_WRAP


@pytest.mark.parametrize("viscous", [False, True])
@pytest.mark.parametrize("P,JM,KM", [(6, 6, 4), (7, 4, 5), (13, 9, 4), (48, 20, 7)])
def test_ogrid_boundaries(P, JM, KM, viscous):
    c = cases.case_naca_ogrid(48, 20, KM, first=2.0e-3, viscous=viscous)
    # a box of the asked size from a ring of the profile's grid: every array wraps
    ring = [np.ascontiguousarray(a[:, :JM, W:W + 48][:, :, np.linspace(0, 47, P).astype(int)]) for a in (c.x, c.y, c.z)]
    c.x, c.y, c.z = (cases.ogrid_wrap(a) if P >= W else a for a in ring)
    c.params["i_end"] = P + 2 * W
    rng = np.random.default_rng(4)
    rho = 1.0 + 0.1 * rng.random((KM + 4, JM + 4, P + 2 * W + 4))
    u, v, w = (0.3 * rng.standard_normal(rho.shape) for _ in range(3))
    c.Q0 = cases.conservative(rho, u, v, w, 1.0 + 0.1 * rng.random(rho.shape), 1.4)
    g, o = pair(c)
    qg = g.get_conservative().reshape(KM + 4, JM + 4, P + 2 * W + 4, 5)
    # wall, k faces, seam: the same sums, products and quotients.  The far field's
    # arithmetic (a power of an entropy) is held by tests/test_gpu_ogrid.py; here
    # its nodes are held to be copied, below
    qo = o.get_conservative().reshape(qg.shape)
    assert rel_linf(qg[:, :JM + 1], qo[:, :JM + 1]) <= 1e-14
    for i in list(range(W + 2)) + list(range(P + W + 2, P + 2 * W + 4)):
        src = i + P if i < W + 2 else i - P
        assert np.array_equal(qg[:, :, i], qg[:, :, src])
    if viscous:
        for a, b in zip(g.get_primitive(), o.get_primitive()):
            a, b = (v.reshape(qg.shape[:3])[:, :JM + 1] for v in (a, b))
            assert rel_linf(a, b) <= 1e-14
