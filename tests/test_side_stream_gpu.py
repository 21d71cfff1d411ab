"""dW* on a stream of its own: gradients are complete for whatever follows backward() on the net's stream, the default one
included, and the products of a weight that two layers share add up."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cnet_b200 import build, configs
from cnet_b200.configs import CROSSENT, FOURIER, GELU, INPUT, LINEAR
from cnet_b200.lib import CnetError
from cnet_b200.net import Net

pytestmark = pytest.mark.gpu


def _train(build, batch, n_in, m, own_stream, captured=False):
    import torch
    net = Net()
    weights = build(net)
    rng = np.random.default_rng(5)
    stream = torch.cuda.Stream() if own_stream else torch.cuda.default_stream()
    net.allocate(batch, stream=stream.cuda_stream if own_stream else None)
    for uid, n, std in weights:
        net.set_values(uid, *[(rng.standard_normal(n) * std).astype(np.float32) for _ in range(2)])
    x = tuple(torch.from_numpy(rng.standard_normal((batch, n_in)).astype(np.float32)).pin_memory() for _ in range(2))
    labels = torch.from_numpy(rng.integers(0, m, batch).astype(np.int32)).pin_memory()
    net.upload(x=x, labels=labels)
    got = []
    with torch.cuda.stream(stream):
        if captured:
            net.sync()
            net.capture_begin()
            net.forward()
            net.backward()
            net.capture_end()
        for _ in range(3):
            net.update_inputs(0.0)                       # clears the gradients
            if captured:
                net.graph_launch()
            else:
                net.forward()
                net.backward()
            got.append(net.grad_tensor().clone())        # in stream order behind backward(), nothing else
    torch.cuda.synchronize()
    net.sync()
    return [g.cpu().numpy() for g in got]


@pytest.mark.parametrize("batch,n", [(128, 128), (300, 500), (260, 1024)])
def test_gradients_are_complete_behind_backward(batch, n):
    def build(net):
        return configs.build_mixer(net, n=n, blocks=3, m=10).weights
    runs = _train(build, batch, n, 10, False) + _train(build, batch, n, 10, True) + _train(build, batch, n, 10, True, captured=True)
    for g in runs[1:]:
        assert np.isfinite(g).all()
        # the same products, perhaps in other schedules: reassociation only
        assert np.linalg.norm(g - runs[0]) < 2e-5 * np.linalg.norm(runs[0])


def test_a_weight_of_two_layers():
    n, m, batch = 128, 10, 128

    def build(net, shared):
        x = net.add(INPUT, n)
        f = net.add(FOURIER, n, prev=[x])
        w = net.add(INPUT, n * n)
        a = net.add(LINEAR, n, n * n, prev=[f, w])
        g = net.add(GELU, n, prev=[a])
        w2 = w if shared else net.add(INPUT, n * n)
        b = net.add(LINEAR, n, n * n, prev=[g, w2])
        wh = net.add(INPUT, n * m)
        head = net.add(LINEAR, n, n * m, prev=[b, wh])
        net.add(CROSSENT, m, prev=[head])
        return [(w, n * n, n ** -0.5)] + ([] if shared else [(w2, n * n, n ** -0.5)]) + [(wh, n * m, n ** -0.5)]

    def grads(shared):
        import torch
        net = Net()
        weights = build(net, shared)
        net.allocate(batch)
        rng = np.random.default_rng(1)
        w = [(rng.standard_normal(n * n) * n ** -0.5).astype(np.float32) for _ in range(2)]
        wh = [(rng.standard_normal(n * m) * n ** -0.5).astype(np.float32) for _ in range(2)]
        for uid, size, _ in weights:
            net.set_values(uid, *(w if size == n * n else wh))
        x = tuple(torch.from_numpy(rng.standard_normal((batch, n)).astype(np.float32)).pin_memory() for _ in range(2))
        net.upload(x=x, labels=torch.from_numpy(rng.integers(0, m, batch).astype(np.int32)).pin_memory())
        for _ in range(2):
            net.update_inputs(0.0)
            net.forward()
            net.backward()
        net.sync()
        return [np.stack(net.get_wgrad(uid)) for uid, size, _ in weights if size == n * n]

    one, two = grads(True), grads(False)
    want = two[0] + two[1]
    assert np.linalg.norm(one[0] - want) < 1e-5 * np.linalg.norm(want)


def _bits(batch, n, how):
    """Gradients of two blocks on a stream of the net's own: launched one by one, captured by the net, or captured by the caller."""
    import torch
    net = Net()
    weights = configs.build_mixer(net, n=n, blocks=2, m=10).weights
    rng = np.random.default_rng(7)
    stream = torch.cuda.Stream()
    net.allocate(batch, stream=stream.cuda_stream)
    for uid, size, std in weights:
        net.set_values(uid, *[(rng.standard_normal(size) * std).astype(np.float32) for _ in range(2)])
    x = tuple(torch.from_numpy(rng.standard_normal((batch, n)).astype(np.float32)).pin_memory() for _ in range(2))
    net.upload(x=x, labels=torch.from_numpy(rng.integers(0, 10, batch).astype(np.int32)).pin_memory())
    net.forward()
    net.backward()
    net.sync()
    with torch.cuda.stream(stream):
        if how == "net":
            net.capture_begin()
            net.forward()
            net.backward()
            net.capture_end()
        elif how == "caller":
            graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            graph.capture_begin(capture_error_mode="thread_local")
            net.forward()
            net.backward()
            graph.capture_end()
        net.update_inputs(0.0)                           # clears the gradients
        if how == "net":
            net.graph_launch()
        elif how == "caller":
            graph.replay()
        else:
            net.forward()
            net.backward()
        got = net.grad_tensor().clone()
    torch.cuda.synchronize()
    net.sync()
    return got.cpu().numpy()


@pytest.mark.parametrize("batch,n", [
    # slices of K without atomics, others on half of the device than on all of it, which the two do not fit on together
    (320, 640),
    (512, 512),
    (1024, 512),
    # what does
    (384, 192),
])
def test_a_nets_own_stream_has_one_schedule(batch, n):
    """Steps that are launched and steps that are replayed, whoever captured them, add up in the same order."""
    runs = [_bits(batch, n, how) for how in ("launched", "net", "caller")]
    assert np.isfinite(runs[0]).all() and (runs[0] == runs[1]).all() and (runs[0] == runs[2]).all()


def test_a_product_that_adds_is_asked_for_as_it_runs():
    """Two layers of one input and one gradient, so that their dW* are the same product.  The second adds its dX* to the first's,
    which is another schedule (512 x 320 -> 512): with it the two products do not fit together, and this dW* runs on half of the
    device, in another order than the other."""
    import torch
    batch, n, m = 512, 320, 512
    net = Net()
    x = net.add(INPUT, n)
    f = net.add(FOURIER, n, prev=[x])
    wa, wb = net.add(INPUT, n * m), net.add(INPUT, n * m)
    a, b = net.add(LINEAR, n, n * m, prev=[f, wa]), net.add(LINEAR, n, n * m, prev=[f, wb])
    s = net.add(configs.RESIDUAL, m, prev=[a, b])
    wh = net.add(INPUT, m * 10)
    net.add(CROSSENT, 10, prev=[net.add(LINEAR, m, m * 10, prev=[s, wh])])
    stream = torch.cuda.Stream()
    net.allocate(batch, stream=stream.cuda_stream)
    rng = np.random.default_rng(2)
    for uid, size in ((wa, n * m), (wb, n * m), (wh, m * 10)):
        net.set_values(uid, *[(rng.standard_normal(size) * n ** -0.5).astype(np.float32) for _ in range(2)])
    planes = tuple(torch.from_numpy(rng.standard_normal((batch, n)).astype(np.float32)).pin_memory() for _ in range(2))
    net.upload(x=planes, labels=torch.from_numpy(rng.integers(0, 10, batch).astype(np.int32)).pin_memory())
    net.forward()
    net.backward()
    net.sync()
    ga, gb = np.stack(net.get_wgrad(wa)), np.stack(net.get_wgrad(wb))
    assert np.linalg.norm(ga - gb) < 1e-5 * np.linalg.norm(ga)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (ga != gb).any()


@pytest.mark.parametrize("join", [0, 1])
def test_an_event_that_fails_is_an_error(join, tmp_path):
    """The second stream is ordered by events alone: a record or a wait that CUDA refuses (of no event) is an error of backward(), also
    where no launch follows that would find it, and nothing is left running on that stream."""
    import torch
    so = str(tmp_path / "probe.so")
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-fno-access-control", "-I/usr/local/cuda/include", os.path.join(here, "cpp", "side_event_probe.cpp"),
                    "-o", so, "-L" + build.HERE, "-l:libcnet_b200.so", "-Wl,-rpath," + build.HERE], check=True)
    swap = C.CDLL(so).swap_side_event
    swap.restype, swap.argtypes = C.c_void_p, [C.c_void_p, C.c_int, C.c_void_p]
    net = Net()
    inp, w, wh = net.add(INPUT, 128), net.add(INPUT, 128 * 128), net.add(INPUT, 1280)
    first = net.add(LINEAR, 128, 128 * 128, prev=[inp, w])               # the last one in backward()
    net.add(CROSSENT, 10, prev=[net.add(LINEAR, 128, 1280, prev=[net.add(GELU, 128, prev=[first]), wh])])
    net.allocate(128)
    rng = np.random.default_rng(3)
    for uid, size in ((w, 128 * 128), (wh, 1280)):
        net.set_values(uid, *[(rng.standard_normal(size) * 0.1).astype(np.float32) for _ in range(2)])
    x = tuple(torch.from_numpy(rng.standard_normal((128, 128)).astype(np.float32)).pin_memory() for _ in range(2))
    net.upload(x=x, labels=torch.zeros(128, dtype=torch.int32).pin_memory())
    net.forward()
    event = swap(net.h, join, None)
    with pytest.raises(CnetError):
        net.backward()
    swap(net.h, join, event)
    torch.cuda.synchronize()
    net.update_inputs(0.0)
    net.forward()
    net.backward()                                       # and with its event again it works
    net.sync()
    assert np.abs(np.stack(net.get_wgrad(w))).max() > 0


def test_a_limit_that_a_caller_has_set_stays():
    """cnb_set_gemm_sm_limit on a net of the default stream: backward() runs under it, and so does what follows."""
    import torch
    batch, n = 512, 512
    runs = []
    for limit in (0, 74):
        net = Net()
        weights = configs.build_mixer(net, n=n, blocks=2, m=10).weights
        net.allocate(batch)
        rng = np.random.default_rng(7)
        for uid, size, std in weights:
            net.set_values(uid, *[(rng.standard_normal(size) * std).astype(np.float32) for _ in range(2)])
        x = tuple(torch.from_numpy(rng.standard_normal((batch, n)).astype(np.float32)).pin_memory() for _ in range(2))
        net.upload(x=x, labels=torch.from_numpy(rng.integers(0, 10, batch).astype(np.int32)).pin_memory())
        assert net.lib.cnb_set_gemm_sm_limit(net.lib.cnh_context(net.h), limit) == 0
        for _ in range(2):                               # the second pass as the first
            net.update_inputs(0.0)
            net.forward()
            net.backward()
            net.sync()
            runs.append(net.grad_tensor().cpu().numpy())
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (runs[0] == runs[1]).all() and (runs[2] == runs[3]).all() and (runs[0] != runs[2]).any()
        assert np.linalg.norm(runs[2] - runs[0]) < 2e-5 * np.linalg.norm(runs[0])
