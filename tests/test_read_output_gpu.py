"""Records read back from a net: what is refused, and batches smaller than the one that was allocated."""
import numpy as np
import pytest

from cnet_b200 import configs
from cnet_b200.net import Net

pytestmark = pytest.mark.gpu


def _net(n, m, allocated, rows):
    net = Net()
    spec = configs.build_classifier(net, n=n, m=m)
    for uid, (re, im) in configs.init_weights(spec, 0).items():
        net.set_values(uid, re, im)
    net.allocate(allocated)
    rng = np.random.default_rng(n)
    x = tuple(rng.standard_normal((rows, n), dtype=np.float32) for _ in range(2))
    net.upload(x=x, labels=np.zeros(rows, np.int32))
    return net, spec, x


def test_a_null_plane_is_refused():
    net, spec, x = _net(64, 10, 8, 3)
    re = np.empty((3, 64), np.float32)
    for a, b in ((None, re.ctypes.data), (re.ctypes.data, None)):
        assert net.lib.cnh_read_output(net.h, spec.main, 0, a, b) < 0
        assert b"null" in net.lib.cnh_error(net.h)
        net.lib.cnh_clear_error(net.h)
    got = net.get_record(spec.main, 0)
    assert np.array_equal(got[0], x[0]) and np.array_equal(got[1], x[1])


@pytest.mark.parametrize("allocated,rows", [(64, 64), (64, 3), (4096, 1)])
def test_part_of_the_allocated_batch(allocated, rows):
    net, spec, x = _net(100, 10, allocated, rows)
    got = net.get_record(spec.main, 0)
    assert np.array_equal(got[0], x[0]) and np.array_equal(got[1], x[1])


def test_planes_further_apart_than_a_copy_may_stride():
    """Planes of 65536 x 8192 floats lie 2^31 bytes apart, one more than the documented limit of a 2D copy's pitch
    (cudaDevAttrMaxPitch; the driver that this was written on takes it all the same)."""
    net = Net()
    spec = configs.build_linear(net, n_in=8192, n_out=2)
    net.allocate(65536)
    x = tuple(np.random.default_rng(1).standard_normal((1, 8192), dtype=np.float32) for _ in range(2))
    net.upload(x=x, labels=np.zeros(1, np.int32))
    got = net.get_record(spec.main, 0)
    assert np.array_equal(got[0], x[0]) and np.array_equal(got[1], x[1])
