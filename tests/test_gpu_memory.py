"""Device memory of a context, from the elements of the padded ghosted box
(csrc/cbns_common.cuh) and the faces.  The limit of the FP32-flux precisions is
what they took before they kept FP32 copies of the state (440 B per node for the
inviscid split): the arrays that the copies make superfluous are not allocated,
so that a block which fitted keeps fitting."""
import pytest
import torch

import cbns3d_cuda_b200 as cb
from cbns3d_cuda_b200 import Block, make_params

pytestmark = pytest.mark.gpu

IM, JM, KM = 256, 256, 64


def _limit(precision, viscous):
    IG, JG, KG = IM + 4, JM + 4, KM + 4
    vol = (13 + IG + 16 + 15) // 16 * 16 * JG * (KG + 1)
    # three state buffers, metrics and Jacobian, area vectors and 1/J, primitives, viscous fluxes and divergence
    need = vol * 8 * (15 + 10 + 10 + 7 + (16 if viscous else 0)) + IG * JG * KG * 40
    if precision != cb.PREC_FP64:
        need += vol * 24 + (10 * IM * JM * KM - 5 * IG * JG * KG) * 8
    if precision == cb.PREC_HYBRID:
        faces = (IM - 1) * (JM - 2) * (KM - 2) + (IM - 2) * (JM - 1) * (KM - 2) + (IM - 2) * (JM - 2) * (KM - 1)
        need += faces * (2 + 32 + 8)
    return need


@pytest.mark.parametrize("precision", [cb.PREC_FP64, cb.PREC_SPLIT, cb.PREC_HYBRID])
@pytest.mark.parametrize("viscous", [False, True])
def test_device_memory_of_a_context(precision, viscous):
    p = make_params(IM, JM, KM, precision=precision, viscous=viscous)
    with Block(p):  # kernels and their tables are loaded once per process
        pass
    free = torch.cuda.mem_get_info()[0]
    with Block(p):
        used = free - torch.cuda.mem_get_info()[0]
    # allocations are rounded up to 2 MB each, about 60 of them
    assert used <= _limit(precision, viscous) + 60 * 2 ** 21
