"""get_record of the layers that run inside a FourierTrans: the values of the batch, also after the weights have moved on."""
import numpy as np
import pytest

import util
from cnet_b200 import configs
from cnet_b200 import lib as L
from cnet_b200.net import Net
from oracle import cnet_oracle as co

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [13, 127, 784, 900, 2048])
def test_hadamard_and_gelu_values(n):
    dev, ora = Net(), co.OracleNet()
    sd, so = configs.build_classifier(dev, n=n, m=5), configs.build_classifier(ora, n=n, m=5)
    for uid, (re, im) in configs.init_weights(sd, 1).items():
        dev.set_values(uid, re, im)
        ora.set_values(uid, re, im)
    dev.allocate(30)
    x, labels = configs.make_batch(sd, 30, 2)
    dev.run_batch(sd.main, x=x, labels=labels)
    ora.run_batch(so.main, x=x, labels=labels)
    dev.update(0.5, 30)
    for name in ("ft", "had", "gelu", "lin"):
        assert util.relerr(dev.get_record(sd.layers[name], 0), ora.get_record(so.layers[name], 0)) < 1e-5, name


@pytest.mark.parametrize("n", [256, 1024, 4096])
def test_products_that_are_never_stored(n):
    net = Net()
    spec = configs.build_classifier(net, n=n, m=5)
    net.allocate(4)
    x, labels = configs.make_batch(spec, 4, 2)
    net.run_batch(spec.main, x=x, labels=labels)
    with pytest.raises(L.CnetError, match="not materialised"):
        net.get_record(spec.layers["had"], 0)
