"""A network whose batch does not fit the device is refused with the library's error, before any host
memory for its batch is asked for, and leaves the process usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_beyond_device_memory_is_refused(fwt):
    from fastweavturb_b200.surrogate import MLP

    with pytest.raises(fwt.FwtError, match="allocation"):
        MLP(n_in=5, width=256, depth=1, n_out=45, batch_max=1 << 30)   # 1 TB of activations in the first layer
    net = MLP(n_in=5, width=64, depth=1, n_out=45, batch_max=64, seed=1)
    assert np.isfinite(net.forward(np.zeros((3, 5), dtype=np.float32))).all()
    net.close()
