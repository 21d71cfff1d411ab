"""The work that users of this library have it do, as cases that can be timed: serving and training steps of the nets
in cnet_b200/configs.py through `Net`, and the operators of `ops.Context` called on torch tensors.

Complex tensors are pairs of float32 planes; there is no other data type on the path.  A training pass is one turn
of the training loop, cut so that the gradients are still there when it ends: update with the gradients of the turn
before, forward, backward, losses on their way to the host.  `prepare` has run the first forward and backward.
"""
import ctypes as C
import math

import torch

from cnet_b200 import configs
from cnet_b200.net import Net
from cnet_b200.ops import Context

LR, BETA = 0.01, 0.9


def listed():
    return [
        # one request of a classifier in service: image in from the host, class scores back to it
        dict(name="classifier_serve_1", kind="serve", net="classifier", batch=1, n=784, m=10),
        # the small classifier's training step as a plain loop calls it: 28 x 28 images, 10 classes
        dict(name="classifier_train_64", kind="train", net="classifier", batch=64, n=784, m=10, update="sgd", graph=False),
        # the same net on 30 x 30 images of 26 letters, a batch that is no power of two, the step captured in a graph
        dict(name="classifier_train_500", kind="train", net="classifier", batch=500, n=900, m=26, update="sgd", graph=True),
        # token-mixing stack: the per-GPU share of a large job, and the whole batch on one GPU (captured steps)
        dict(name="mixer_train_512", kind="train", net="mixer", batch=512, n=1024, blocks=8, m=10, update="sgd", graph=True),
        dict(name="mixer_train_4096", kind="train", net="mixer", batch=4096, n=1024, blocks=8, m=10, update="sgd", graph=True),
        # a smaller stack at a width that is no power of two, trained with Adam (which cannot be captured)
        dict(name="mixer_adam_300", kind="train", net="mixer", batch=300, n=500, blocks=4, m=10, update="adam", graph=False),
        # embedding language model: training step, and the loss of a last, partial batch of an evaluation
        dict(name="lm_train_1024", kind="train", net="lm", batch=1024, tokens=64, vocab=8192, dim=256, hidden=2048,
             update="sgd", graph=False),
        dict(name="lm_eval_100", kind="eval", net="lm", batch=100, tokens=64, vocab=8192, dim=256, hidden=2048),
        # one Linear layer, forward and both backward products, called as operators: square, and ragged in every size
        dict(name="linear_4096", kind="linear", batch=4096, n_in=4096, n_out=4096),
        dict(name="linear_777", kind="linear", batch=777, n_in=1333, n_out=1001),
        # FourierTrans forward and backward on a batch of signals, at a length with no factor beyond 2, 3 and 5
        dict(name="fourier_1500", kind="fourier", batch=1000, n=1500),
        # a classification head: normalised scores, loss and its gradient back to the scores
        dict(name="loss_1000", kind="loss", batch=4096, m=1000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """One more case: the nets and operators above at sizes spread over the range that they are used in."""
    kind = rng.choice(["serve", "classifier", "classifier", "mixer", "mixer", "lm", "eval", "linear", "linear", "fourier",
                       "fourier", "loss"])
    if kind == "serve":
        return dict(kind="serve", net="classifier", batch=_log_int(rng, 1, 256), n=_log_int(rng, 64, 2048), m=rng.randint(2, 100))
    if kind == "classifier":
        graph = rng.random() < 0.5
        return dict(kind="train", net="classifier", batch=_log_int(rng, 16, 2048), n=_log_int(rng, 64, 2048),
                    m=rng.randint(2, 100), update="sgd" if graph else rng.choice(["sgd", "adam"]), graph=graph)
    if kind == "mixer":
        n = rng.choice([64, 128, 256, 512, 1024, _log_int(rng, 64, 1024), _log_int(rng, 64, 1024)])
        blocks = rng.randint(1, 8)
        batch = _log_int(rng, 64, max(64, min(4096, (1 << 32) // (n * n * blocks))))
        graph = rng.random() < 0.5
        return dict(kind="train", net="mixer", batch=batch, n=n, blocks=blocks, m=rng.randint(2, 100),
                    update="sgd" if graph else rng.choice(["sgd", "adam"]), graph=graph)
    if kind in ("lm", "eval"):
        c = dict(net="lm", batch=_log_int(rng, 16, 1024), tokens=rng.randint(8, 64), vocab=_log_int(rng, 256, 8192),
                 dim=_log_int(rng, 16, 256), hidden=_log_int(rng, 64, 2048))
        return dict(c, kind="eval") if kind == "eval" else dict(c, kind="train", update="sgd", graph=rng.random() < 0.5)
    if kind == "linear":
        return dict(kind="linear", batch=_log_int(rng, 16, 4096), n_in=_log_int(rng, 16, 4096), n_out=_log_int(rng, 4, 4096))
    if kind == "fourier":
        n = rng.choice([64, 128, 256, 512, 1024, 2048, 4096, _log_int(rng, 32, 4096), _log_int(rng, 32, 4096)])
        return dict(kind="fourier", batch=_log_int(rng, 1, max(1, (1 << 22) // n)), n=n)
    m = _log_int(rng, 10, 32768)
    return dict(kind="loss", batch=_log_int(rng, 1, max(1, min(65536, (1 << 23) // m))), m=m)


# ------------------------------------------------------------------------------------------------- preparation
def _builder(case):
    if case["net"] == "classifier":
        return configs.build_classifier, dict(n=case["n"], m=case["m"])
    if case["net"] == "mixer":
        return configs.build_mixer, dict(n=case["n"], blocks=case["blocks"], m=case["m"])
    return configs.build_embed_lm, dict(tokens=case["tokens"], vocab=case["vocab"], dim=case["dim"], hidden=case["hidden"])


def _planes(gen, *shape, std=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * std, torch.randn(*shape, generator=gen, device="cuda") * std)


def _batch(case, spec, gen):
    """A batch on the host, pinned, with the distributions of cnet_b200/configs.py, and its labels."""
    b = case["batch"]
    labels = torch.randint(0, spec.n_classes, (b,), generator=gen, device="cuda", dtype=torch.int32).cpu().pin_memory()
    if spec.tokens:
        tok = torch.randint(0, spec.vocab, (b, spec.in_dim), generator=gen, device="cuda", dtype=torch.int32)
        return dict(tokens=tok.cpu().pin_memory(), labels=labels)
    if spec.name == "classifier":                          # images: real parts uniform, no imaginary part
        re = torch.rand(b, spec.in_dim, generator=gen, device="cuda")
        im = torch.zeros_like(re)
    else:
        re, im = _planes(gen, b, spec.in_dim)
    return dict(x=(re.cpu().pin_memory(), im.cpu().pin_memory()), labels=labels)


def _weight_view(net):
    """All weights of the net, as the device holds them: one float32 range of its arena."""
    p, n = C.c_void_p(), C.c_size_t()
    net.lib.cnh_weight_arena(net.h, C.byref(p), C.byref(n))
    off = p.value - net.arena.data_ptr()
    return net.arena[off:off + 4 * n.value].view(torch.float32)


class State:
    pass


_stream = None


def _capturable_stream():
    """The stream of the captured steps, one for the whole program: a captured step cannot run on the default one."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream.cuda_stream


def _update(s):
    if s.case["update"] == "adam":
        s.net.adam_update(LR / s.case["batch"], BETA, s.t)
        s.t += 1
    else:
        s.net.update_inputs(LR / s.case["batch"])


def prepare(case, seed):
    s = State()
    s.case = case
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if "net" in case:
        build, sizes = _builder(case)
        s.net = Net()
        s.spec = build(s.net, **sizes)
        for uid, n, std in s.spec.weights:
            re, im = _planes(gen, n, std=std)
            s.net.set_values(uid, re.cpu().numpy(), im.cpu().numpy())
        s.net.allocate(case["batch"], stream=_capturable_stream() if case.get("graph") else None)
        s.host = _batch(case, s.spec, gen)
        s.losses = torch.empty(case["batch"], pin_memory=True)
        s.net.upload(**s.host)
        if case["kind"] == "train":
            s.t = 0
            s.net.forward()
            s.net.backward()
            if case["graph"]:
                _update(s)
                s.net.forward()
                s.net.backward()
                s.net.sync()
                s.net.capture_begin()
                _update(s)
                s.net.forward()
                s.net.backward()
                s.net.capture_end()
            s.weights, s.grads = _weight_view(s.net), s.net.grad_tensor()
        s.net.sync()
        return s
    if case["kind"] == "linear":
        b, i, o = case["batch"], case["n_in"], case["n_out"]
        s.ctx = Context(arena_bytes=(64 << 20) + 40 * (b * i + b * o + i * o))     # operand copies of every product
        s.x, s.w, s.g = _planes(gen, b, i, std=i ** -0.5), _planes(gen, o, i, std=i ** -0.5), _planes(gen, b, o)
    elif case["kind"] == "fourier":
        b, n = case["batch"], case["n"]
        s.ctx = Context(arena_bytes=(64 << 20) + 48 * n * n + 48 * b * n)          # tables and operand copies
        s.x, s.g = _planes(gen, b, n), _planes(gen, b, n)
    else:
        s.ctx = Context(arena_bytes=64 << 20)
        s.z = _planes(gen, case["batch"], case["m"])
        s.labels = torch.randint(0, case["m"], (case["batch"],), generator=gen, device="cuda", dtype=torch.int32)
    return s


# -------------------------------------------------------------------------------------------------------- pass
def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "serve":
        s.net.upload(**s.host)
        s.net.infer()
        return s.net.get_record(s.spec.layers["lin"], 0)
    if kind == "eval":
        s.net.infer()
        s.net.read_losses_async(s.losses, case["batch"])
        return s.losses
    if kind == "train":
        if case["graph"]:
            s.net.graph_launch()
        else:
            _update(s)
            s.net.forward()
            s.net.backward()
        s.net.read_losses_async(s.losses, case["batch"])
        return s.losses, s.grads, s.weights
    if kind == "linear":
        return s.ctx.linear_fwd(s.x, s.w), s.ctx.linear_bwd_x(s.g, s.w), s.ctx.linear_bwd_w(s.g, s.x)
    if kind == "fourier":
        return s.ctx.dft_fwd(s.x), s.ctx.dft_bwd(s.g)
    y, inv = s.ctx.softmax_fwd(s.z)
    loss, d = s.ctx.crossent(y, s.labels)
    return loss, y, s.ctx.softmax_bwd(d, s.z, inv)


# ------------------------------------------------------------------------------------------- least work, tolerance
def _fourier_flops(b, n):
    return 5.0 * b * n * math.log2(n)


def work(case):
    b = case["batch"]
    if case["kind"] == "linear":
        i, o = case["n_in"], case["n_out"]
        return {"bytes": 8.0 * 2 * (b * i + o * i + b * o), "flops": 3 * 8.0 * b * i * o}
    if case["kind"] == "fourier":
        return {"bytes": 8.0 * 4 * b * case["n"], "flops": 2 * _fourier_flops(b, case["n"])}
    if case["kind"] == "loss":
        return {"bytes": 8.0 * 3 * b * case["m"] + 8.0 * b, "flops": 24.0 * b * case["m"]}
    # nets: the batch, the weights and what is returned; activations need not leave the chip
    build, sizes = _builder(case)
    if case["net"] == "lm":
        d = case["tokens"] * case["dim"]
        linear = [(d, case["hidden"]), (case["hidden"], case["vocab"])]
        weights = case["vocab"] * case["dim"]
        fourier, x_bytes = 0.0, 4.0 * b * case["tokens"]
    else:
        n, blocks = case["n"], case.get("blocks", 1)
        linear = ([(n, n)] * blocks if case["net"] == "mixer" else []) + [(n, case["m"])]
        weights = n * blocks
        fourier, x_bytes = blocks * _fourier_flops(b, n), 8.0 * b * n
    flops = fourier + sum(8.0 * b * i * o for i, o in linear)
    weights += sum(i * o for i, o in linear)
    if case["kind"] == "serve":
        return {"bytes": x_bytes + 8.0 * weights + 8.0 * b * case["m"], "flops": flops}
    if case["kind"] == "eval":
        if case["net"] == "lm":                            # of the table, the rows that the tokens name
            weights += min(0, b * case["tokens"] - case["vocab"]) * case["dim"]
        return {"bytes": x_bytes + 8.0 * weights + 8.0 * b, "flops": flops}
    # weights and gradients (and Adam's momentum) are read and written once each
    per_weight = 8.0 * (6 if case["update"] == "adam" else 4)
    return {"bytes": x_bytes + per_weight * weights + 8.0 * b, "flops": 3 * flops}


def tolerance(case):
    """Everything is computed in float32 or in splits that keep about 20 bits.  A sum of products differs by some 1e-5
    between orders of summation; through the layers of a net, forward and back, by a few times that."""
    if case["kind"] in ("fourier", "loss"):
        return {"rel": 1e-5}
    if case["kind"] == "linear":
        return {"rel": 2e-5}
    return {"rel": 1e-4}
