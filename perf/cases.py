"""Performance cases: the training and evaluation work that programs hand to this backend, over the sizes it is used at.

Two ways in are used, the ones the README shows. A *run* goes through `omb.Trainer`: a number of training steps replayed
from the captured step, each on a batch of its own that was staged from pinned host memory one step ahead, then a read of
the updated parameters (what a program that keeps its best weights does once per interval). A *step* goes through the tensor
and module API: forward, loss, backward and optimizer called one by one. An *eval* is a forward pass without a tape.

A parameter whose gradient is zero in exact arithmetic (a bias in front of a batch norm, an attention key's bias) gets rounding
noise instead: no output consists of such values alone.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "onemodel-csharp_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import om_binding as omb  # noqa: E402

TIERS = {"fp32": 0, "tf32": omb.OM_TF32, "bf16": omb.OM_TF32 | omb.OM_BF16_OPERANDS}
_ctx = None


def context(flags):
    """The process's one device context, with the flags of the case at hand."""
    global _ctx
    if _ctx is None:
        _ctx = omb.Context(0, flags)
    if _ctx.flags != flags:
        _ctx.set_flags(flags)
    return _ctx


def flags_of(case):
    # The recurrent layers' time steps in one cooperative launch each: what bench.py uses for the recurrent configuration.
    return TIERS[case["tier"]] | (omb.OM_SEQ_KERNELS if case["kind"] == "crnn-run" else 0)


def listed():
    return [
        # The smallest call: one step of a small classifier in the exact fp32 tier through the module API; host work and
        # launches are what it costs.
        {"name": "mlp-step-small-fp32", "kind": "mlp-step", "tier": "fp32", "batch": 16, "in": 64, "hidden": 128, "out": 10},
        # The MLP configuration (784-512-512-10, batch 128): a launch-bound captured step.
        {"name": "mlp-run", "kind": "mlp-run", "tier": "tf32", "batch": 128, "in": 784, "hidden": 512, "out": 10, "steps": 16},
        # The CNN configuration: eight 3x3 convolutions with batch norm on 256 images of 32x32, SGD with momentum.
        {"name": "cnn-run", "kind": "cnn-run", "tier": "tf32", "batch": 256, "in": 3, "height": 32, "width": 32, "classes": 10,
         "channels": "64,64,128,128,256,256,512,512", "strides": "1,1,2,1,2,1,2,1", "steps": 4},
        # A user's own small CNN on images of an odd size with a ragged batch and channel counts off the tile sizes.
        {"name": "cnn-step-ragged", "kind": "cnn-step", "tier": "tf32", "batch": 37, "in": 3, "height": 45, "width": 51,
         "classes": 17, "channels": 24},
        # The text-line recogniser configuration: convolutions, two bidirectional LSTM layers, CTC, Adam.
        {"name": "crnn-run", "kind": "crnn-run", "tier": "tf32", "batch": 64, "height": 32, "width": 256, "classes": 97, "hidden": 256,
         "max_label": 20, "channels": "64,128,256,256", "steps": 4},
        # The MiniLM-shape encoder configuration (TF32 products, sequences of one attention tile).
        {"name": "minilm-run", "kind": "encoder-run", "tier": "tf32", "batch": 64, "seq": 128, "layers": 6, "width": 384, "heads": 12,
         "ff": 1536, "vocab": 30522, "rows": 1229, "steps": 8},
        # The BERT-base-shape encoder configuration (bfloat16 products, sequences of several attention tiles): the largest.
        {"name": "bert-run", "kind": "encoder-run", "tier": "bf16", "batch": 32, "seq": 512, "layers": 12, "width": 768, "heads": 12,
         "ff": 3072, "vocab": 30522, "rows": 2458, "steps": 8},
        # A small encoder whose batch, sequence and vocabulary are off every tile size, bfloat16 products.
        {"name": "encoder-run-ragged", "kind": "encoder-run", "tier": "bf16", "batch": 7, "seq": 201, "layers": 3, "width": 320, "heads": 5,
         "ff": 1280, "vocab": 5003, "rows": 211, "steps": 8},
        # Fine-tuning a classifier over padded sequences with a mask through the tensor API (TF32 products).
        {"name": "encoder-step-masked", "kind": "encoder-step", "tier": "tf32", "batch": 16, "seq": 320, "layers": 3, "width": 256, "heads": 8,
         "ff": 1024, "vocab": 8192, "classes": 5},
        # Scoring masked positions with a trained encoder: forward only, logits over the whole vocabulary, bfloat16 products.
        {"name": "encoder-eval", "kind": "encoder-eval", "tier": "bf16", "batch": 32, "seq": 256, "layers": 4, "width": 512, "heads": 8,
         "ff": 2048, "vocab": 30522, "rows": 1229},
    ]


def _log(rng, low, high):
    """A whole number from [low, high], evenly spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["mlp-step", "mlp-run", "cnn-run", "cnn-step", "crnn-run", "encoder-run", "encoder-run", "encoder-step", "encoder-eval"])
    if kind == "mlp-step":
        return {"kind": kind, "tier": rng.choice(["fp32", "tf32"]), "batch": _log(rng, 4, 512), "in": _log(rng, 16, 1024), "hidden": _log(rng, 32, 1024),
                "out": _log(rng, 2, 100)}
    if kind == "mlp-run":
        return {"kind": kind, "tier": rng.choice(["tf32", "bf16"]), "batch": _log(rng, 32, 4096), "in": _log(rng, 64, 1024), "hidden": 8 * _log(rng, 16, 256),
                "out": _log(rng, 2, 1000), "steps": 16}
    if kind == "cnn-run":
        base, side = 8 * rng.randint(2, 8), rng.randint(20, 40)
        channels = [base, base, 2 * base, 2 * base, 4 * base, 4 * base][: rng.choice([4, 6])]
        strides = [1, 1, 2, 1, 2, 1][: len(channels)]
        return {"kind": kind, "tier": "tf32", "batch": _log(rng, 16, 256), "in": rng.choice([1, 3]), "height": side, "width": side + rng.randint(0, 12),
                "classes": rng.randint(2, 100), "channels": ",".join(map(str, channels)), "strides": ",".join(map(str, strides)), "steps": 4}
    if kind == "cnn-step":
        return {"kind": kind, "tier": "tf32", "batch": _log(rng, 8, 128), "in": rng.choice([1, 3]), "height": rng.randint(24, 64), "width": rng.randint(24, 64),
                "classes": rng.randint(2, 100), "channels": 4 * rng.randint(4, 16)}
    if kind == "crnn-run":
        c = 16 * rng.randint(1, 4)
        return {"kind": kind, "tier": "tf32", "batch": _log(rng, 8, 64), "height": 32, "width": 4 * rng.randint(30, 80), "classes": rng.randint(30, 120),
                "hidden": 32 * rng.randint(2, 8), "max_label": rng.randint(8, 12), "channels": "%d,%d,%d,%d" % (c, 2 * c, 4 * c, 4 * c), "steps": 4}
    head = rng.choice([32, 64])
    heads = rng.randint(4, 12)
    width = head * heads
    tokens = _log(rng, 512, 16384)
    seq = rng.randint(48, 512)
    batch = max(1, tokens // seq)
    case = {"kind": kind, "tier": rng.choice(["tf32", "bf16"]), "batch": batch, "seq": seq, "layers": rng.randint(1, 4), "width": width, "heads": heads,
            "ff": 4 * width, "vocab": _log(rng, 1000, 30522)}
    if kind == "encoder-step":
        case["layers"], case["classes"] = min(3, case["layers"]), rng.randint(2, 20)
    else:
        case["rows"] = max(1, batch * seq * 15 // 100)
    if kind == "encoder-run":
        case["steps"] = 4
    return case


# ---- runs through the trainers --------------------------------------------------------------------------------------------
def _ints(text):
    return [int(v) for v in text.split(",")]


def _trainer(case, seed):
    # A tenth of the configurations' learning rates, as late in a schedule: what rounding changes then stays small over a pass.
    k = case["kind"]
    if k == "mlp-run":
        return omb.Trainer("mlp", [case["batch"], case["in"], case["hidden"], case["hidden"], case["out"]], lr=1e-4, weight_decay=0.01, seed=seed)
    if k == "cnn-run":
        ch, st = _ints(case["channels"]), _ints(case["strides"])
        return omb.Trainer("cnn", [case["batch"], case["in"], case["height"], case["width"], case["classes"], len(ch)] + ch + st, lr=0.01, weight_decay=0.0,
                           seed=seed)
    if k == "crnn-run":
        return omb.Trainer("crnn", [case["batch"], case["height"], case["width"], case["classes"], case["hidden"], case["max_label"]] + _ints(case["channels"]),
                           lr=1e-4, weight_decay=0.0, seed=seed)
    return omb.Trainer("mlm", [case[n] for n in ("batch", "seq", "layers", "width", "heads", "ff", "vocab", "rows")], lr=1e-5, weight_decay=0.01, seed=seed)


def _batch(case, rng):
    """One host batch, with the distributions of the benchmark configurations."""
    k, b = case["kind"], case["batch"]
    if k == "mlp-run":
        return [rng.standard_normal((b, case["in"]), dtype=np.float32), rng.integers(0, case["out"], b)]
    if k == "cnn-run":
        return [rng.standard_normal((b, case["in"], case["height"], case["width"]), dtype=np.float32), rng.integers(0, case["classes"], b)]
    if k == "crnn-run":
        lengths = rng.integers(5, case["max_label"] + 1, b).astype(np.int32)
        targets = np.zeros(b * case["max_label"], np.int32)
        targets[: int(lengths.sum())] = rng.integers(1, case["classes"], int(lengths.sum()))
        return [rng.random((b, 1, case["height"], case["width"]), dtype=np.float32), targets, lengths]
    ids = rng.integers(0, case["vocab"], (b, case["seq"])).astype(np.int32)
    rows = np.sort(rng.choice(b * case["seq"], case["rows"], replace=False)).astype(np.int32)
    return [ids, rows, ids.reshape(-1)[rows].astype(np.int64)]


class _Run:
    """A trainer with its captured step, the pinned host batches of the coming steps and the pinned memory parameters are read into."""

    def __init__(self, case, seed):
        self.flags = flags_of(case)
        context(self.flags)
        rng = np.random.default_rng(seed)
        self.trainer = _trainer(case, seed)
        for _ in range(2):   # eager steps fill the memory pool the capture draws from
            self.trainer.step(_batch(case, rng))
        self.trainer.enable_graph()
        self.trainer.prefetch_depth(2)
        self.pinned = [[torch.from_numpy(a).pin_memory() for a in _batch(case, rng)] for _ in range(case["steps"])]
        self.tables = [(C.c_void_p * len(b))(*[t.data_ptr() for t in b]) for b in self.pinned]
        self.losses = torch.zeros(case["steps"], dtype=torch.float32)
        # The parameters of one module lie behind one another, those of the same module of every layer too: parameters[module][layer].
        groups = {}
        for i, (name, shape) in enumerate(self.trainer.named_parameters()):
            module, _, _ = name.rpartition(".")
            kind = ".".join(p for p in module.split(".") if not p.isdigit()) if module.startswith("layers.") else module
            groups.setdefault(kind, {}).setdefault(module, []).append((i, math.prod(shape)))
        self.parameters, self.targets = {}, []
        for kind, modules in groups.items():
            out = torch.zeros((len(modules), sum(n for _, n in next(iter(modules.values())))), dtype=torch.float32, pin_memory=True)
            self.parameters[kind] = out
            for row, members in zip(out, modules.values()):
                at = 0
                for i, n in members:
                    self.targets.append((C.c_int32(i), C.c_void_p(row[at:].data_ptr())))
                    at += n

    def __call__(self):
        context(self.flags)
        tr, n = self.trainer, len(self.tables)
        loss = C.c_float()
        tr.prefetch_ptrs(self.tables[0])
        for i in range(n):
            if i + 1 < n:
                tr.prefetch_ptrs(self.tables[i + 1])
            tr.step_prefetched(C.byref(loss))
            self.losses[i] = loss.value
        lib = omb.host_lib()
        for i, where in self.targets:
            omb.Trainer._check(lib.omh_trainer_get_param(tr.h, i, where))
        return {"losses": self.losses, "parameters": self.parameters}

    def __del__(self):
        tr = getattr(self, "trainer", None)
        if tr is not None:
            tr.close()
            _ctx.call("om_pool_trim", _ctx.handle)


# ---- steps through the tensor and module API ------------------------------------------------------------------------------
class _Memory:
    """Device memory of a tensor under the CUDA array interface (keeps the tensor alive)."""

    def __init__(self, t):
        self.tensor = t
        self.__cuda_array_interface__ = {"shape": tuple(t.shape), "typestr": "<f4", "data": (t.data_ptr, False), "version": 2}


def view(t):
    return torch.as_tensor(_Memory(t), device="cuda")


def _parameter(rng, shape, bound):
    return omb.Tensor.from_numpy(((2 * rng.random(shape, dtype=np.float32) - 1) * np.float32(bound)).astype(np.float32), requires_grad=True)


class _Encoder:
    """Token and position embeddings and post-norm encoder layers, written against the tensor API."""

    def __init__(self, case, rng, head_width):
        d, ff = case["width"], case["ff"]
        self.case, self.p = case, {}

        def linear(name, i, o):
            self.p[name + ".weight"], self.p[name + ".bias"] = _parameter(rng, (o, i), i ** -0.5), _parameter(rng, (o,), i ** -0.5)

        def norm(name):
            self.p[name + ".weight"] = omb.Tensor.from_numpy(np.ones(d, np.float32), requires_grad=True)
            self.p[name + ".bias"] = omb.Tensor.from_numpy(np.zeros(d, np.float32), requires_grad=True)

        self.p["tok"], self.p["pos"] = _parameter(rng, (case["vocab"], d), 1.0), _parameter(rng, (case["seq"], d), 1.0)
        for i in range(case["layers"]):
            for n in "qkvo":
                linear("%d.%s" % (i, n), d, d)
            norm("%d.norm1" % i)
            linear("%d.ff1" % i, d, ff)
            linear("%d.ff2" % i, ff, d)
            norm("%d.norm2" % i)
        linear("head", d, head_width)
        self.positions = omb.Tensor.from_numpy(np.arange(case["seq"], dtype=np.int32))

    def linear(self, name, x):
        return omb.call("linear", [x, self.p[name + ".weight"], self.p[name + ".bias"]])

    def __call__(self, ids, mask=None):
        p, call, heads = self.p, omb.call, self.case["heads"]
        x = call("add", [call("embedding", [p["tok"], ids]), call("embedding", [p["pos"], self.positions])])
        for i in range(self.case["layers"]):
            n = "%d." % i
            q, k, v = (self.linear(n + c, x) for c in "qkv")
            a = self.linear(n + "o", call("attention_heads", [q, k, v, mask], ints=[heads]))
            x = call("add_layer_norm", [x, a, p[n + "norm1.weight"], p[n + "norm1.bias"]])
            f = call("feed_forward", [x, p[n + "ff1.weight"], p[n + "ff1.bias"], p[n + "ff2.weight"], p[n + "ff2.bias"]])
            x = call("add_layer_norm", [x, f, p[n + "norm2.weight"], p[n + "norm2.bias"]])
        return x


class _Step:
    """One training step called operation by operation: the gradients and the updated state are what it leaves."""

    def __init__(self, case, seed):
        self.flags = flags_of(case)
        context(self.flags)
        rng = np.random.default_rng(seed)
        if case["kind"] == "encoder-step":
            parameters = self._encoder(case, rng)
            self.optimizer = omb.Optimizer.adamw(list(parameters.values()), 1e-4)
        else:
            parameters = self._modules(case, rng, seed)
            if case["kind"] == "mlp-step":
                self.optimizer = omb.Optimizer.adamw(list(parameters.values()), 1e-3)
            else:
                self.optimizer = omb.Optimizer.sgd(list(parameters.values()), 0.05, momentum=0.9)
        self.outputs = {}
        self()               # a program's first step: the gradients get their memory, which later steps write again
        for name, t in parameters.items():
            if case["kind"] != "cnn-step" and not name.endswith("k.bias"):
                self.outputs["gradient." + name] = view(t.grad)
            if case["kind"] == "mlp-step":
                self.outputs["weight." + name] = view(t)
        if case["kind"] == "cnn-step":   # (its gradients pass through ReLU and pooling decisions that any rounding can flip)
            self.outputs.update(("state." + name, view(t)) for name, t in self.model.state_dict())

    def _modules(self, case, rng, seed):
        M, g = omb.Module, omb.Generator(seed)
        b = case["batch"]
        if case["kind"] == "mlp-step":
            h = case["hidden"]
            self.model = M.sequential(M("linear", g, [case["in"], h, 1]), M("relu"), M("linear", g, [h, h, 1]), M("relu"), M("linear", g, [h, case["out"], 1]))
            x, classes = rng.standard_normal((b, case["in"]), dtype=np.float32), case["out"]
        else:
            c = case["channels"]
            block = lambda i, o, pool: [M("conv2d", g, [i, o, 3, 1, 1, 1]), M("batch_norm2d", ints=[o]), M("relu"), pool]  # noqa: E731
            self.model = M.sequential(*block(case["in"], c, M("max_pool2d", ints=[2, 2, 0])), *block(c, 2 * c, M("max_pool2d", ints=[2, 2, 0])),
                                      *block(2 * c, 4 * c, M("global_avg_pool2d")), M("flatten"), M("linear", g, [4 * c, case["classes"], 1]))
            x, classes = rng.standard_normal((b, case["in"], case["height"], case["width"]), dtype=np.float32), case["classes"]
            for name, t in self.model.named_parameters():   # the norms of a network that has been trained for a while
                if len(t.shape) == 1 and name.endswith("weight"):
                    t.copy_from(rng.uniform(0.5, 1.5, t.shape))
                elif name in ("1.bias", "5.bias", "9.bias"):
                    t.copy_from(0.2 * rng.standard_normal(t.shape))
        self.x, self.y = omb.Tensor.from_numpy(x), omb.Tensor.from_numpy(rng.integers(0, classes, b))
        self.forward = lambda: self.model(self.x)
        return dict(self.model.named_parameters())

    def _encoder(self, case, rng):
        b, l = case["batch"], case["seq"]
        net = _Encoder(case, rng, case["classes"])
        self.ids = omb.Tensor.from_numpy(rng.integers(0, case["vocab"], (b, l)).astype(np.int32))
        self.y = omb.Tensor.from_numpy(rng.integers(0, case["classes"], b))
        lengths = rng.integers(max(1, l // 2), l + 1, b)   # padded keys are masked out with a large negative score
        padded = np.where(np.arange(l)[None, :] < lengths[:, None], 0.0, -1e9).astype(np.float32)
        self.mask = omb.Tensor.from_numpy(np.repeat(padded[:, None, :], l, axis=1))
        self.forward = lambda: net.linear("head", omb.call("select", [net(self.ids, self.mask)], ints=[1, 0]))
        return net.p

    def __call__(self):
        context(self.flags)
        logits = self.forward()
        loss = omb.call("cross_entropy", [logits, self.y])
        self.optimizer.zero_grad()
        loss.backward()
        self.optimizer.step()
        return dict(self.outputs, loss=view(loss), logits=view(logits))


class _Eval:
    """Logits of the masked positions of one batch."""

    def __init__(self, case, seed):
        self.flags = flags_of(case)
        context(self.flags)
        rng = np.random.default_rng(seed)
        self.net = _Encoder(case, rng, case["vocab"])
        b, l = case["batch"], case["seq"]
        self.tokens, self.width = b * l, case["width"]
        self.ids = omb.Tensor.from_numpy(rng.integers(0, case["vocab"], (b, l)).astype(np.int32))
        self.rows = omb.Tensor.from_numpy(np.sort(rng.choice(b * l, case["rows"], replace=False)).astype(np.int32))

    def __call__(self):
        context(self.flags)
        with omb.no_grad():
            x = self.net(self.ids)
            picked = omb.call("embedding", [x.reshape(self.tokens, self.width), self.rows])
            logits = self.net.linear("head", picked)
        return {"logits": view_rows(logits)}


def view_rows(t):
    """A rank-2 view of rows that may lie further apart than they are long."""
    _, shape, strides = t._info()
    m = _Memory(t)
    m.__cuda_array_interface__ = dict(m.__cuda_array_interface__, strides=tuple(4 * s for s in strides))
    return torch.as_tensor(m, device="cuda")


def prepare(case, seed):
    if case["kind"].endswith("-run"):
        return _Run(case, seed)
    return _Eval(case, seed) if case["kind"] == "encoder-eval" else _Step(case, seed)


def run(state):
    return state()


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def _encoder_work(case, head):
    """(parameters, forward flops) of an encoder whose head maps `head` rows."""
    d, ff, n, l = case["width"], case["ff"], case["batch"] * case["seq"], case["seq"]
    out = case["classes"] if "classes" in case else case["vocab"]
    params = (case["vocab"] + l) * d + case["layers"] * (4 * d * d + 2 * d * ff + 9 * d + ff) + out * (d + 1)
    flops = case["layers"] * (2 * n * (4 * d * d + 2 * d * ff) + 4 * n * l * d) + 2 * head * d * out
    return params, flops


def _conv_work(case):
    """(parameters, forward flops) of the convolutional configurations."""
    k, b = case["kind"], case["batch"]
    h, w, c, params, flops = case["height"], case["width"], case.get("in", 1), 0, 0
    if k == "cnn-step":
        channels, strides, pools = [case["channels"] * f for f in (1, 2, 4)], [1, 1, 1], [(2, 2), (2, 2), (1, 1)]
    elif k == "cnn-run":
        channels, strides = _ints(case["channels"]), _ints(case["strides"])
        pools = [(1, 1)] * len(channels)
    else:
        channels, strides, pools = _ints(case["channels"]), [1] * 4, [(2, 2), (2, 2), (2, 1), (4, 1)]
    for o, s, (ph, pw) in zip(channels, strides, pools):
        h, w = (h - 1) // s + 1, (w - 1) // s + 1
        flops += 2 * b * h * w * o * c * 9
        params += o * c * 9 + (o if k == "crnn-run" else 3 * o)
        h, w, c = h // ph, w // pw, o
    if k == "crnn-run":
        t, hid = w, case["hidden"]
        for i in (c, 2 * hid):
            params += 2 * 4 * hid * (i + hid + 2)
            flops += 2 * 2 * t * b * 4 * hid * (i + hid)
        c, b = 2 * hid, t * b
    params += (c + 1) * case["classes"]
    return params, flops + 2 * b * c * case["classes"]


def work(case):
    k, b = case["kind"], case["batch"]
    if k.startswith("mlp"):
        sizes = [case["in"], case["hidden"], case["hidden"], case["out"]]
        params = sum((i + 1) * o for i, o in zip(sizes, sizes[1:]))
        flops, inputs = 2 * b * sum(i * o for i, o in zip(sizes, sizes[1:])), 4 * b * case["in"] + 8 * b
    elif k.startswith("encoder"):
        params, flops = _encoder_work(case, case.get("rows", b))
        inputs = 4 * b * case["seq"] + (12 * case["rows"] if "rows" in case else 8 * b)
        if k == "encoder-step":
            inputs += 4 * b * case["seq"] ** 2
    else:
        params, flops = _conv_work(case)
        inputs = 4 * b * case.get("in", 1) * case["height"] * case["width"] + 8 * b
    if k == "encoder-eval":   # the rows of the token table that the batch names, the other weights, the logits
        rows = min(case["vocab"], b * case["seq"])
        return {"bytes": 4 * (params - (case["vocab"] - rows) * case["width"]) + inputs + 4 * case["rows"] * case["vocab"], "flops": flops}
    # A training step reads and writes the weights and the optimizer's moments, and writes the gradients once.
    state = 20 if k.startswith("cnn") else 28
    steps = case.get("steps", 1)
    return {"bytes": steps * (inputs + state * params), "flops": 3 * steps * flops}


# About four times what a relative change of 5e-7 in the starting weights (what another order of the sums does) was seen to do
# over two passes of the listed and forty drawn cases: {kind: {tier: (rel, max)}}. Where a rounded operand falls on the other
# side, a product moves by a step of its operand type; Adam's first steps turn the sign of a near-zero gradient into a whole
# step of the learning rate, which sets the largest single differences.
TOLERANCES = {
    "mlp-step": {"fp32": (1e-3, 5e-2), "tf32": (8e-3, 0.2)},
    "mlp-run": {"tf32": (5e-3, 0.1), "bf16": (5e-3, 0.1)},
    "cnn-run": {"tf32": (2.5e-3, 2e-2)},
    "cnn-step": {"tf32": (1.5e-3, 2e-2)},
    "crnn-run": {"tf32": (4e-3, 0.35)},
    "encoder-run": {"tf32": (2e-4, 1.2e-2), "bf16": (4e-4, 3e-2)},
    "encoder-step": {"tf32": (7e-3, 0.1), "bf16": (2e-2, 0.45)},
    "encoder-eval": {"tf32": (8e-4, 5e-3), "bf16": (6.5e-3, 4e-2)},
}


def tolerance(case):
    rel, most = TOLERANCES[case["kind"]][case["tier"]]
    return {"rel": rel, "max": most}
