"""Predictions on both sides of the sizes where the outputs leave their standardisation on the
host or on the device: the same bits as numpy's."""
import numpy as np
import pytest

from indicatrix_b200 import surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members,m", [(1, 1), (1, 255), (1, 256), (2, 1), (2, 31), (2, 32), (3, 9), (3, 10), (4, 3), (4, 4)])
def test_predictions_equal_numpy(members, m):
    ens = surrogate.SurrogateEnsemble(members, seed=11)
    rng = np.random.default_rng(members * 1000 + m)
    for net in ens.nets:
        net.t_std = rng.uniform(0.1, 9.0, 27).astype(np.float32)
        net.t_mean = rng.standard_normal(27).astype(np.float32)
    x = surrogate.normalize(surrogate.sample_designs(m, m))
    xb = ens.nets[0].to_device_bf16(x)
    want = np.stack([net.forward_device(xb)[0].cpu().numpy() * net.t_std + net.t_mean for net in ens.nets])
    before = surrogate.launches
    got = ens.predict_members(x)
    on_device = m * members ** 3 >= 256
    # One conversion, four layers a member, and a scaling launch a member on the device.
    assert surrogate.launches - before == 1 + members * (5 if on_device else 4)
    assert got.dtype == want.dtype and got.flags.writeable and np.array_equal(got, want)
    assert np.array_equal(ens.nets[0].predict(x), want[0])
