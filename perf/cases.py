"""The work that programs written against this framework have it do, as a list of measurable cases.

Every case is one call of a function that ``cgt_b200.function`` compiled: a training step (forward, ``cgt.grad``
backward, parameter update), a prediction, or one step of a recurrent network that generates. A training step returns
the loss and every variable it updates (weights, biases, optimizer slots), as views of the device memory where the
framework keeps them; a prediction returns the arrays that the call returns.

Fields that all kinds share: ``batch``; ``data``: where the caller's arrays are, "host" (plain numpy arrays, as
scripts pass them) or "device" (``runtime.device_array``, a data set that stays on the GPU).
"""
import numpy as np
import torch

import cgt_b200 as cgt
from cgt_b200 import configs, nn, runtime

KINDS = ("mlp_predict", "mlp_train", "convnet_predict", "convnet_train", "wide_train", "lstm_train", "lstm_step", "vae_train")


def listed():
    return [
        # one example at a time through a small classifier, as a service answers requests: latency only
        dict(name="mlp_predict_one", kind="mlp_predict", batch=1, xdim=784, hidden=256, classes=10, precision="single",
             free_batch=False, data="host"),
        # the MLP configuration's training step at its own batch, from host arrays as a digit-recognition script passes
        # them; the batch extent is left open so that the last, shorter batch of an epoch goes through the same function
        dict(name="mlp_train_b128", kind="mlp_train", batch=128, xdim=784, hidden=256, classes=10, precision="single",
             free_batch=True, data="host"),
        # the same step in double precision, as gradient checks and small scientific fits run it
        dict(name="mlp_train_double", kind="mlp_train", batch=100, xdim=200, hidden=120, classes=10, precision="double",
             free_batch=False, data="host"),
        # large dense layers and a large batch: the step is made of large products
        dict(name="mlp_train_large", kind="mlp_train", batch=2048, xdim=1024, hidden=3072, classes=100, precision="single",
             free_batch=False, data="device"),
        # the CIFAR-shape convnet, the headline configuration
        dict(name="convnet_train_b128", kind="convnet_train", batch=128, image=32, channels=3, filters1=32, filters2=32, filters3=64,
             kernel=5, pool=3, lrn=True, classes=10, data="device"),
        # a smaller network on one-channel images: filter counts and batch that are not multiples of anything
        dict(name="convnet_train_gray", kind="convnet_train", batch=50, image=28, channels=1, filters1=20, filters2=50, filters3=50,
             kernel=3, pool=2, lrn=False, classes=10, data="host"),
        # evaluation of the CIFAR-shape network on a test set, a few hundred images per call
        dict(name="convnet_predict_b500", kind="convnet_predict", batch=500, image=32, channels=3, filters1=32, filters2=32, filters3=64,
             kernel=5, pool=3, lrn=True, classes=10, data="host"),
        # the wide convolution stack's share of one GPU
        dict(name="wide_train_b128", kind="wide_train", batch=128, data="device"),
        # the two-layer character-level LSTM configuration, unrolled over 50 characters
        dict(name="lstm_train_t50", kind="lstm_train", batch=64, vocab=65, hidden=128, layers=2, seq_len=50, data="host"),
        # a short unrolling with odd sizes, one layer
        dict(name="lstm_train_t15", kind="lstm_train", batch=33, vocab=47, hidden=90, layers=1, seq_len=15, data="host"),
        # the trained LSTM generates text, one character per call, the state handed from call to call
        dict(name="lstm_step_one", kind="lstm_step", batch=1, vocab=65, hidden=128, layers=2, data="host"),
        # the variational autoencoder configuration, Adam updates
        dict(name="vae_train_b100", kind="vae_train", batch=100, xdim=784, hidden=500, zdim=20, data="host"),
    ]


def _log_int(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(KINDS)
    data = rng.choice(("host", "device"))
    if kind == "mlp_predict":
        return dict(kind=kind, batch=_log_int(rng, 1, 1024), xdim=_log_int(rng, 32, 1024), hidden=_log_int(rng, 32, 1024),
                    classes=rng.randint(2, 100), precision=rng.choice(("single", "single", "single", "double")),
                    free_batch=rng.random() < 0.3, data=data)
    if kind == "mlp_train":
        if rng.random() < 0.2:
            return dict(kind=kind, batch=_log_int(rng, 16, 256), xdim=_log_int(rng, 32, 784), hidden=_log_int(rng, 32, 256),
                        classes=rng.randint(2, 100), precision="double", free_batch=rng.random() < 0.3, data=data)
        return dict(kind=kind, batch=_log_int(rng, 16, 2048), xdim=_log_int(rng, 32, 1024), hidden=_log_int(rng, 32, 3072),
                    classes=rng.randint(2, 100), precision="single", free_batch=rng.random() < 0.3, data=data)
    if kind in ("convnet_predict", "convnet_train"):
        image, pool = rng.choice(((28, 2), (32, 2), (32, 3), (32, 3)))
        return dict(kind=kind, batch=_log_int(rng, 1, 400) if kind == "convnet_predict" else _log_int(rng, 16, 128),
                    image=image, channels=rng.choice((1, 3, 3)), filters1=rng.choice((16, 20, 32, 32)),
                    filters2=rng.choice((32, 32, 48, 50)), filters3=rng.choice((32, 50, 64, 64)), kernel=rng.choice((3, 5)),
                    pool=pool, lrn=rng.random() < 0.5, classes=rng.randint(2, 100), data=data)
    if kind == "wide_train":
        return dict(kind=kind, batch=_log_int(rng, 8, 128), data=data)
    if kind == "lstm_train":
        return dict(kind=kind, batch=_log_int(rng, 8, 64), vocab=rng.randint(30, 100), hidden=rng.choice((32, 50, 64, 90, 100, 128)),
                    layers=rng.choice((1, 2)), seq_len=_log_int(rng, 5, 50), data=data)
    if kind == "lstm_step":
        return dict(kind=kind, batch=_log_int(rng, 1, 64), vocab=rng.randint(30, 100), hidden=_log_int(rng, 32, 512),
                    layers=rng.choice((1, 2)), data=data)
    return dict(kind=kind, batch=_log_int(rng, 16, 512), xdim=_log_int(rng, 64, 784), hidden=_log_int(rng, 64, 1000),
                zdim=rng.randint(2, 50), data=data)


# ------------------------------------------------------------------------------------------------
# networks, written as user scripts write them
# ------------------------------------------------------------------------------------------------
def _loss(logits, y):
    logprobs = nn.logsoftmax(logits)
    return -logprobs[cgt.arange(cgt.size(logits, 0)), y].mean()


def _mlp(case):
    batch = None if case["free_batch"] else case["batch"]
    X = cgt.matrix("X", fixed_shape=(batch, case["xdim"]))
    y = cgt.vector("y", dtype="i8", fixed_shape=(batch,))
    sizes = (case["xdim"], case["hidden"], case["hidden"])
    h = X
    for i in range(2):
        h = cgt.tanh(nn.Affine(sizes[i], sizes[i + 1], name="fc%d" % i, weight_init=nn.XavierNormal())(h))
    return X, y, nn.Affine(sizes[2], case["classes"], name="out", weight_init=nn.XavierNormal())(h)


def _pooled(size, pool):
    return -(-(size - pool) // 2)


def _convnet(case):
    n, k = case["image"], case["kernel"]
    X = cgt.tensor4("X", fixed_shape=(case["batch"], case["channels"], n, n))
    y = cgt.vector("y", dtype="i8", fixed_shape=(case["batch"],))
    he = nn.HeNormal(scale=float(np.sqrt(2.0)))
    h, c = X, case["channels"]
    for i in (1, 2, 3):
        conv = nn.SpatialConvolution(c, case["filters%d" % i], kernelshape=(k, k), pad=(k // 2, k // 2), name="conv%d" % i, weight_init=he)
        h = nn.max_pool_2d(nn.rectify(conv(h)), kernelshape=(case["pool"], case["pool"]), stride=(2, 2))
        if i == 1 and case["lrn"]:
            h = nn.cross_channel_lrn(h, 5, 1e-4, 0.75)
        c, n = case["filters%d" % i], _pooled(n, case["pool"])
    d0, d1, d2, d3 = h.shape
    flat = h.reshape([d0, d1 * d2 * d3])
    return X, y, nn.Affine(c * n * n, case["classes"], name="ip", weight_init=nn.HeNormal(scale=1.0))(flat)


def _cell(x, h, c, x2h, h2h, hidden):
    sums = x2h(x) + h2h(h)
    gates = cgt.sigmoid(sums[:, 0:3 * hidden])
    c = gates[:, hidden:2 * hidden] * c + gates[:, 0:hidden] * cgt.tanh(sums[:, 3 * hidden:4 * hidden])
    return gates[:, 2 * hidden:3 * hidden] * cgt.tanh(c), c


def _lstm_step(case):
    """Function of (x, h_0, c_0, ...) -> probabilities and new states, or, when the data stay on the GPU, of (x) ->
    probabilities with the states as shared variables that the call updates."""
    B, H = case["batch"], case["hidden"]
    init = nn.IIDUniform(-0.3, 0.3)
    x = cgt.matrix("x", fixed_shape=(B, case["vocab"]))
    args, states, news = [x], [], []
    out, size = x, case["vocab"]
    for i in range(case["layers"]):
        if case["data"] == "device":
            h, c = (cgt.shared(np.zeros((B, H), "f4"), fixed_shape_mask="all") for _ in range(2))
            states += [h, c]
        else:
            h, c = (cgt.matrix(name, fixed_shape=(B, H)) for name in ("h", "c"))
            args += [h, c]
        x2h = nn.Affine(size, 4 * H, name="l%d.x2h" % i, weight_init=init)
        h2h = nn.Affine(H, 4 * H, name="l%d.h2h" % i, weight_init=init)
        out, c_new = _cell(out, h, c, x2h, h2h, H)
        news += [out, c_new]
        size = H
    probs = nn.softmax(nn.Affine(H, case["vocab"], name="pred", weight_init=init)(out))
    return args, probs, states, news


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
class _View(object):
    """Device memory of a shared variable for torch (CUDA array interface); keeps the memory alive."""

    def __init__(self, variable):
        self.owner = variable.op._value
        self.__cuda_array_interface__ = dict(shape=tuple(self.owner.shape), typestr="<" + self.owner.dtype,
                                             data=(self.owner.data, False), version=3)


def _views(updates):
    return [torch.as_tensor(_View(before), device="cuda") for (before, _after) in updates]


def _arguments(case, arrays):
    return [runtime.device_array(a) for a in arrays] if case["data"] == "device" else list(arrays)


def _one_hot(rs, n, classes):
    return np.eye(classes, dtype="f4")[rs.randint(0, classes, size=n)]


def _train(X, y, logits, lr):
    loss = _loss(logits, y)
    updates = nn.sgd(loss, nn.get_parameters(loss), lr)
    return cgt.function([X, y], [loss], updates=updates), updates


def prepare(case, seed):
    kind, B = case["kind"], case["batch"]
    rs = np.random.RandomState(seed)
    np.random.seed(seed)  # the layers draw their weights from numpy's global generator
    updates = []
    if kind in ("mlp_predict", "mlp_train"):
        with cgt.scoped_update_config(precision=case["precision"]):
            X, y, logits = _mlp(case)
            if kind == "mlp_predict":
                f = cgt.function([X], [nn.softmax(logits)])
            else:
                f, updates = _train(X, y, logits, 0.01)
            arrays = [rs.rand(B, case["xdim"]).astype(cgt.floatX), rs.randint(0, case["classes"], size=B).astype("i8")]
    elif kind in ("convnet_predict", "convnet_train"):
        X, y, logits = _convnet(case)
        if kind == "convnet_predict":
            f = cgt.function([X], [nn.softmax(logits)])
        else:
            f, updates = _train(X, y, logits, 0.001)
        arrays = [rs.randn(B, case["channels"], case["image"], case["image"]).astype("f4"),
                  rs.randint(0, case["classes"], size=B).astype("i8")]
    elif kind == "lstm_step":
        args, probs, states, news = _lstm_step(case)
        H = case["hidden"]
        if case["data"] == "device":
            updates = list(zip(states, news))
            f = cgt.function(args, [probs], updates=updates)
            for s in states:
                s.op.set_value((rs.randn(B, H) * 0.5).astype("f4"))
            arrays = [_one_hot(rs, B, case["vocab"])]
        else:
            f = cgt.function(args, [probs] + news)
            arrays = [_one_hot(rs, B, case["vocab"])] + [(rs.randn(B, H) * 0.5).astype("f4") for _ in range(2 * case["layers"])]
    else:
        if kind == "wide_train":
            cfg = configs.build_wide(batch=B, seed=seed)
        elif kind == "lstm_train":
            cfg = configs.build_lstm(vocab=case["vocab"], hidden=case["hidden"], n_layers=case["layers"], seq_len=case["seq_len"],
                                     batch=B, seed=seed)
        else:
            cfg = configs.build_vae(batch=B, xdim=case["xdim"], hdim=case["hidden"], zdim=case["zdim"], seed=seed)
        f, updates, arrays = cfg.compile(), cfg.updates, cfg.batch(seed + 1)
    if kind.endswith("_predict"):
        arrays = arrays[:1]
    return dict(f=f, args=_arguments(case, arrays), vars=_views(updates), carry=kind == "lstm_step" and case["data"] == "host")


def run(state):
    outs = state["f"](*state["args"])
    if state["carry"]:  # the new states are the next call's arguments
        state["args"] = state["args"][:1] + outs[1:]
    return outs + state["vars"]


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _dense(sizes, batch, train):
    """(parameters, flops) of dense layers of the given sizes; a training step multiplies three times per layer, twice
    in the first one, whose input needs no gradient."""
    pairs = list(zip(sizes[:-1], sizes[1:]))
    params = sum((a + 1) * b for (a, b) in pairs)
    macs = sum(a * b for (a, b) in pairs)
    return params, 2.0 * batch * ((3 * macs - pairs[0][0] * pairs[0][1]) if train else macs)


def _conv(batch, pixels, cin, cout, k, passes):
    return (cin * k * k + 1) * cout, 2.0 * passes * batch * pixels * cin * k * k * cout


def work(case):
    """Bytes: inputs and weights read once, results and updated variables written once. Flops: the products and
    convolutions."""
    kind, B = case["kind"], case["batch"]
    size = 4
    if kind in ("mlp_predict", "mlp_train"):
        train = kind == "mlp_train"
        size = 8 if case["precision"] == "double" else 4
        params, flops = _dense((case["xdim"], case["hidden"], case["hidden"], case["classes"]), B, train)
        values = B * case["xdim"] + (2 * params if train else params + B * case["classes"])
    elif kind in ("convnet_predict", "convnet_train"):
        train = kind == "convnet_train"
        n, c, params, flops = case["image"], case["channels"], 0, 0.0
        for i in (1, 2, 3):
            p, fl = _conv(B, n * n, c, case["filters%d" % i], case["kernel"], (2 if i == 1 else 3) if train else 1)
            params, flops, c, n = params + p, flops + fl, case["filters%d" % i], _pooled(n, case["pool"])
        p = (c * n * n + 1) * case["classes"]
        params, flops = params + p, flops + 2.0 * (3 if train else 1) * B * p
        values = B * case["channels"] * case["image"] ** 2 + (2 * params if train else params + B * case["classes"])
    elif kind == "wide_train":
        p1, f1 = _conv(B, 15 * 15, 3, 96, 11, 2)
        p2, f2 = _conv(B, 6 * 6, 96, 256, 5, 3)
        p3, f3 = _dense((1024, 4096, 100), B, True)
        flops = f1 + f2 + f3 + 2.0 * B * 1024 * 4096
        values = B * 3 * 64 * 64 + 2 * (p1 + p2 + p3)
    elif kind in ("lstm_train", "lstm_step"):
        H, V, T = case["hidden"], case["vocab"], case.get("seq_len", 1)
        macs = sum(((V if i == 0 else H) + H) * 4 * H for i in range(case["layers"])) + H * V
        params = macs + 8 * H * case["layers"] + V
        train = kind == "lstm_train"
        flops = 2.0 * (3 if train else 1) * B * T * macs
        values = 2 * params + 2 * T * B * V if train else params + 2 * B * V + 4 * case["layers"] * B * H
    else:
        p1, f1 = _dense((case["xdim"], case["hidden"], 2 * case["zdim"]), B, True)
        p2, f2 = _dense((case["zdim"], case["hidden"], case["xdim"]), B, True)
        flops = f1 + f2 + 2.0 * B * case["zdim"] * case["hidden"]
        values = B * (case["xdim"] + case["zdim"]) + 6 * (p1 + p2)
    return {"bytes": float(size * values), "flops": float(flops)}


def tolerance(case):
    """Largest relative errors of another correct implementation of the same precision."""
    if case.get("precision") == "double":
        return {"rel": 1e-11, "max": 1e-9}
    if case["kind"] == "vae_train":
        # Adam's first steps divide a gradient by its own magnitude: where rounding decides the sign of a gradient that is
        # all but zero, that weight moves by twice the step, a fifth of the weights' root mean square
        return {"rel": 1e-3, "max": 0.5}
    # 32-bit sums; the biases start at zero and hold a gradient that cancels over the batch, and a pooling window or a
    # rectifier whose arguments tie to within rounding sends single terms of it elsewhere
    return {"rel": 2e-5 if case["kind"].endswith(("_predict", "_step")) else 1e-4, "max": 1e-2}
