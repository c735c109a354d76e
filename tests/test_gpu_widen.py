"""The widening of the sensor's decisions on its bit rows, at line lengths on
both sides of a 32-face word and at the smallest and largest widths.

Decisions are whole numbers: the widened set equals the dense widening of the
predictor's decisions on the sampled features, up to faces that a decision
within 1e-4 of the threshold can change."""
import numpy as np
import pytest

from cbns3d_cuda_b200 import CBNS_Q, PREC_HYBRID, Block, cases, make_params
from tests.test_gpu_hybrid import _flat

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from cbns3d_cuda_b200 import sensor  # noqa: E402


def _widen(dec, shape, along, across):
    """Dense widening, windows larger than the block included."""
    IM, JM, KM = shape
    out, at = [], 0
    for own, n in ((2, (KM - 2, JM - 2, IM - 1)), (1, (KM - 2, JM - 1, IM - 2)), (0, (KM - 1, JM - 2, IM - 2))):
        r = dec[at:at + n[0] * n[1] * n[2]].reshape(n)
        at += r.size
        for ax in range(3):
            w, src = (along if ax == own else across), np.moveaxis(r, ax, 0)
            r = np.moveaxis(np.stack([src[max(0, x - w):x + w + 1].max(axis=0) for x in range(n[ax])]), 0, ax)
        out.append(r.reshape(-1))
    return np.concatenate(out)


@pytest.mark.parametrize("every", [1, 8])
@pytest.mark.parametrize("shape", [(12, 9, 9), (33, 12, 9), (34, 9, 12), (35, 21, 10), (66, 14, 11), (131, 12, 23)])
def test_widened_decisions(shape, every):
    c = cases.case_shock_vortex(*shape)
    h = Block(make_params(*c.shape, **c.params, precision=PREC_HYBRID))
    h.calc_metrics(c.x, c.y, c.z)
    h.set_conservative(c.Q0)
    h.set_bc_calc_primitive(CBNS_Q)
    # logit = (sum |f| - cut) / cut, cut at the strongest 3% of the faces
    X, _y, _d, idx = sensor.sample_faces(h, with_dev=True)
    s = np.abs(X.cpu().numpy().astype(np.float64)).sum(axis=1)
    P = np.zeros(sensor.NPARAM, dtype=np.float32)
    for m in range(sensor.NIN):
        P[sensor.P_W1 + (2 * m) * sensor.NIN + m] = 1.0
        P[sensor.P_W1 + (2 * m + 1) * sensor.NIN + m] = -1.0
    P[sensor.P_W2:sensor.P_W2 + 2 * sensor.NIN] = 1.0
    P[sensor.P_W3] = 1.0 / float(np.quantile(s, 0.97))
    P[sensor.P_B3] = -1.0
    h.sensor_load(P, 0.5)
    h.sensor_audit(97, 1.0e30)
    h.sensor_interval(every)
    h.sensor_stats_reset()
    h.set_time(0.0)
    assert h.run(1) == 1  # decisions of the initial state
    got, forced = h.sensor_mask()
    p = sensor.predict(torch.from_numpy(P).cuda(), X, tensor_cores=True).cpu().numpy()
    idx = idx.cpu().numpy()
    near, want = np.zeros(got.size, bool), np.zeros(got.size, np.uint8)
    near[idx] = np.abs(p - 0.5) < 1e-4
    want[idx] = (p >= 0.5) & ~_flat(X)
    lo, hi = (_widen(w, c.shape, 1 + every, every) for w in (want & ~near, want | near))
    assert not forced and 0 < want.sum() < want.size
    assert np.all((got >= lo) & (got <= hi))
    assert h.sensor_stats()["weno_faces"] == int(got.sum())
