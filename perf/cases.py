"""Performance cases of the spectral path: what programs written on this package have it do.

Kinds of work, with the place in this repository their sizes come from:

  classify   the spherical classifier S2Conv -> ReLU -> SO3Conv -> ReLU -> so3_integrate -> Linear
             (``models.S2ConvNet_original``, the network of ``bench.py``): inference through ``fuse``,
             called eagerly or replayed as a CUDA graph, and training
  deep       ``models.S2ConvNet_deep``: seven convolutions at full bandwidth 30 and below, with batch
             normalisation in the head: inference and training
  shape      the wide multi-channel shape classifier (bandwidths 64 -> 16 -> 10 -> 5, 6 -> 100 -> 100
             -> 255 channels, the training step of ``bench.py``): inference and training
  layer      one SO3Convolution, forward and backward (also with odd channel counts and bandwidths)
  so3        one direction of the SO(3) transform on its own, from the small bandwidths of the tests to
             the b = 64 of ``bench.py``, also between two bandwidths
  s2         the S2 transforms, analysis then synthesis
  rotate     ``so3_rotation`` of a batch of signals by an arbitrary rotation (augmentation, equivariance
             checks)

Everything is float32, the only type the package takes.
"""
import math

import numpy as np
import torch

import s2cnn_b200 as S
from s2cnn_b200.graph import GraphedForward
from s2cnn_b200.soft.s2_fft import S2_fft_real, S2_ifft_real
from s2cnn_b200.soft.so3_fft import so3_rfft, so3_rifft


def listed():
    return [
        # one image arrives at a time: the latency of an answer, called as plain Python
        {"name": "classify one", "kind": "classify", "mode": "infer", "batch": 1, "graph": False,
         "f1": 20, "f2": 40, "b_in": 30, "b_l1": 10, "b_l2": 6},
        # throughput inference at the batch size of bench.py, captured as a graph
        {"name": "classify batch", "kind": "classify", "mode": "infer", "batch": 256, "graph": True,
         "f1": 20, "f2": 40, "b_in": 30, "b_l1": 10, "b_l2": 6},
        # the classifier's training step at the batch size of the reference's example
        {"name": "classify train", "kind": "classify", "mode": "train", "batch": 32, "graph": False,
         "f1": 20, "f2": 40, "b_in": 30, "b_l1": 10, "b_l2": 6},
        # the deep network on the last, incomplete batch of a test set
        {"name": "deep ragged", "kind": "deep", "mode": "infer", "batch": 7, "bandwidth": 30},
        # the deep network's training step
        {"name": "deep train", "kind": "deep", "mode": "train", "batch": 32, "bandwidth": 30},
        # the wide network's training step: the largest contractions
        {"name": "shape train", "kind": "shape", "mode": "train", "batch": 32,
         "b0": 64, "b1": 16, "b2": 10, "b3": 5, "f0": 6, "f1": 100, "f2": 100, "f3": 255},
        # a small layer with odd channel counts and bandwidths, forward and backward
        {"name": "layer odd", "kind": "layer", "batch": 5, "f_in": 13, "f_out": 9, "b_in": 11, "b_out": 7},
        # the transform benchmark, each direction on its own
        {"name": "so3 analysis 64", "kind": "so3", "direction": "analysis", "batch": 64, "b": 64, "b_spec": 64},
        {"name": "so3 synthesis 64", "kind": "so3", "direction": "synthesis", "batch": 64, "b": 64, "b_spec": 64},
        # a bandwidth that is no power of two, an odd number of signals, some degrees dropped
        {"name": "so3 analysis 22", "kind": "so3", "direction": "analysis", "batch": 45, "b": 22, "b_spec": 15},
        # images on the sphere to spectra and back, six channels of the shape classifier's grid
        {"name": "s2 round trip", "kind": "s2", "batch": 192, "b": 64, "b_spec": 64},
        # random rotation of a batch of signals
        {"name": "rotate", "kind": "rotate", "batch": 32, "features": 8, "b": 12},
    ]


def _log_int(rng, lo, hi):
    """A whole number of lo .. hi, spread over its logarithm."""
    return int(min(hi, max(lo, math.floor(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _bandwidth(rng, lo, hi):
    """A bandwidth of lo .. hi, spread over its logarithm.  The transforms take lengths whose prime
    factors are at most 31."""
    while True:
        b = _log_int(rng, lo, hi)
        if b <= 31 or all(b % p for p in (37, 41, 43, 47, 53, 59, 61)):
            return b


def draw(rng):
    kind = rng.choice(["classify", "classify", "deep", "shape", "layer", "so3", "so3", "s2", "rotate"])
    if kind == "classify":
        mode = rng.choice(["infer", "infer", "train"])
        b_l1 = rng.randint(6, 14)
        return {"kind": kind, "mode": mode, "graph": mode == "infer" and rng.random() < 0.5,
                "batch": _log_int(rng, 1 if mode == "infer" else 4, 256 if mode == "infer" else 64),
                "f1": rng.randint(10, 32), "f2": rng.randint(20, 48), "b_in": rng.randint(20, 32),
                "b_l1": b_l1, "b_l2": rng.randint(4, min(8, b_l1))}
    if kind == "deep":
        return {"kind": kind, "mode": rng.choice(["infer", "train"]), "batch": _log_int(rng, 2, 32),
                "bandwidth": rng.randint(16, 30)}
    if kind == "shape":
        return {"kind": kind, "mode": rng.choice(["infer", "train"]), "batch": _log_int(rng, 2, 32),
                "b0": rng.choice([32, 48, 64]), "b1": rng.randint(12, 16), "b2": rng.randint(7, 10),
                "b3": rng.randint(3, 5), "f0": rng.choice([3, 6]), "f1": rng.randint(40, 100),
                "f2": rng.randint(40, 100), "f3": rng.randint(60, 255)}
    if kind == "layer":
        b_in = rng.randint(4, 16)
        return {"kind": kind, "batch": _log_int(rng, 1, 64), "f_in": _log_int(rng, 4, 64),
                "f_out": _log_int(rng, 4, 64), "b_in": b_in, "b_out": rng.randint(3, min(b_in, 12))}
    if kind == "so3":
        b = rng.choice([_bandwidth(rng, 4, 48), 32, 64])
        most = max(1, int(64 * (64 / b) ** 3))
        return {"kind": kind, "direction": rng.choice(["analysis", "synthesis"]),
                "batch": _log_int(rng, 1, min(4096, most)), "b": b,
                "b_spec": b if rng.random() < 0.5 else rng.randint(max(2, b // 3), b)}
    if kind == "s2":
        b = _bandwidth(rng, 8, 64)
        return {"kind": kind, "batch": _log_int(rng, 1, 512), "b": b,
                "b_spec": b if rng.random() < 0.5 else rng.randint(max(4, b // 4), b)}
    return {"kind": "rotate", "batch": _log_int(rng, 1, 64), "features": rng.randint(1, 20), "b": rng.randint(4, 20)}


# ------------------------------------------------------------------------------------------------
# the programs
# ------------------------------------------------------------------------------------------------
class _Shape(torch.nn.Module):
    """The wide shape classifier, written as a user of the reference writes it."""

    def __init__(self, c):
        super().__init__()
        g2, g3 = _shape_grids()
        self.c1 = S.S2Convolution(c["f0"], c["f1"], c["b0"], c["b1"], g2)
        self.c2 = S.SO3Convolution(c["f1"], c["f2"], c["b1"], c["b2"], g3)
        self.c3 = S.SO3Convolution(c["f2"], c["f3"], c["b2"], c["b3"], g3)
        self.lin = torch.nn.Linear(c["f3"], 55)

    def forward(self, x):
        x = torch.relu(self.c1(x))
        x = torch.relu(self.c2(x))
        x = torch.relu(self.c3(x))
        return self.lin(S.so3_integrate(x))


def _shape_grids():
    return (S.s2_near_identity_grid(max_beta=np.pi / 32, n_alpha=8, n_beta=3),
            S.so3_near_identity_grid(max_beta=np.pi / 8, max_gamma=2 * np.pi, n_alpha=8, n_beta=3, n_gamma=8))


def _model(c):
    if c["kind"] == "classify":
        return S.models.S2ConvNet_original(f1=c["f1"], f2=c["f2"], b_in=c["b_in"], b_l1=c["b_l1"], b_l2=c["b_l2"])
    if c["kind"] == "deep":
        return S.models.S2ConvNet_deep(bandwidth=c["bandwidth"])
    return _Shape(c)


def _input_shape(c):
    if c["kind"] == "classify":
        return (c["batch"], 1, 2 * c["b_in"], 2 * c["b_in"])
    if c["kind"] == "deep":
        return (c["batch"], 1, 2 * c["bandwidth"], 2 * c["bandwidth"])
    return (c["batch"], c["f0"], 2 * c["b0"], 2 * c["b0"])


def prepare(case, seed):
    c = dict(case)
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(seed)
    torch.manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device=dev)

    if c["kind"] in ("classify", "deep", "shape"):
        model = _model(c)
        with torch.no_grad():
            for name, p in model.named_parameters():
                if name.endswith("bias"):
                    p.normal_(0, 0.1)          # biases start at zero; a network in use has others
        model = model.to(dev).train(c["mode"] == "train")
        st = {"what": c["mode"], "x": randn(*_input_shape(c))}
        # a network written with plain calls, handed to fuse(); the classifier trains as it is written
        st["model"] = model if c["kind"] == "classify" and c["mode"] == "train" else S.fuse(model)
        if c["mode"] == "train":
            st["labels"] = torch.randint(0, 55 if c["kind"] == "shape" else 10, (c["batch"],), generator=gen, device=dev)
        elif c.get("graph"):
            st["model"] = GraphedForward(st["model"], st["x"])
        return st
    if c["kind"] == "layer":
        g3 = S.so3_near_identity_grid(max_beta=np.pi / 8, max_gamma=2 * np.pi, n_alpha=8, n_beta=3, n_gamma=8)
        n, m = 2 * c["b_in"], 2 * c["b_out"]
        return {"what": "layer", "model": S.SO3Convolution(c["f_in"], c["f_out"], c["b_in"], c["b_out"], g3).to(dev),
                "x": randn(c["batch"], c["f_in"], n, n, n).requires_grad_(True),
                "gy": randn(c["batch"], c["f_out"], m, m, m)}
    n = 2 * c["b"]
    if c["kind"] == "so3":
        if c["direction"] == "analysis":
            return {"what": "analysis", "x": randn(c["batch"], n, n, n), "b_out": c["b_spec"]}
        return {"what": "synthesis", "x": so3_spectrum(c["batch"], c["b_spec"], randn), "b_out": c["b"]}
    if c["kind"] == "s2":
        return {"what": "s2", "x": randn(c["batch"], n, n), "b": c["b"], "b_spec": c["b_spec"]}
    rng = np.random.RandomState(seed % (1 << 32))
    return {"what": "rotate", "x": randn(c["batch"], c["features"], n, n, n),
            "angles": [float(v) for v in rng.uniform(0, 1, 3) * np.array([2 * np.pi, np.pi, 2 * np.pi])]}


def so3_spectrum(batch, b, randn):
    """Random spectrum of real signals, [l * m * n, batch, complex]: X[l,-m,-n] = (-1)^(m-n) conj X[l,m,n]."""
    rows = []
    for l in range(b):
        x = torch.view_as_complex(randn(2 * l + 1, 2 * l + 1, batch, 2))
        k = torch.arange(-l, l + 1, device=x.device)
        sign = (1 - 2 * ((k[:, None] - k[None, :]).abs() % 2)).view(2 * l + 1, 2 * l + 1, 1)
        rows.append(torch.view_as_real((x + sign * x.flip(0, 1).conj()) / 2).reshape(-1, batch, 2))
    return torch.cat(rows).contiguous()


def run(state):
    what = state["what"]
    if what == "infer":
        if isinstance(state["model"], GraphedForward):
            return state["model"](state["x"])
        with torch.no_grad():
            return state["model"](state["x"])
    if what == "train":
        model = state["model"]
        model.zero_grad(set_to_none=True)
        loss = torch.nn.functional.cross_entropy(model(state["x"]), state["labels"])
        loss.backward()
        out = {"loss": loss.detach()}
        out.update(("grad " + k, p.grad) for k, p in model.named_parameters())
        out.update(("buffer " + k, b) for k, b in model.named_buffers() if b.is_floating_point())
        return out
    if what == "layer":
        model, x = state["model"], state["x"]
        model.zero_grad(set_to_none=True)
        x.grad = None
        y = model(x)
        y.backward(state["gy"])
        return {"y": y.detach(), "gx": x.grad, "gkernel": model.kernel.grad, "gbias": model.bias.grad}
    if what == "analysis":
        return so3_rfft(state["x"], b_out=state["b_out"])
    if what == "synthesis":
        return so3_rifft(state["x"], b_out=state["b_out"])
    if what == "s2":
        spec = S2_fft_real.apply(state["x"], state["b_spec"])
        return {"spectrum": spec, "signal": S2_ifft_real.apply(spec, state["b"])}
    return S.so3_rotation(state["x"], *state["angles"])


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _n3(b):
    return b * (4 * b * b - 1) // 3


def _so3_flops(signals, b, k):
    """One SO(3) transform of real signals: 2-D FFTs of the planes, then the Wigner contraction of the
    Hermitian half of the coefficients over beta."""
    n = 2 * b
    return signals * (n * 2.5 * n * n * math.log2(n * n) + 2.0 * _n3(k) * n)


def _s2_flops(signals, b, k):
    n = 2 * b
    return signals * (2.5 * n * n * math.log2(n) + 2.0 * k * k * n)


def _net_layers(c):
    """(f_in, f_out, b_in, b_out, grid points) of every convolution, the S2 one first."""
    if c["kind"] == "classify":
        return [(1, c["f1"], c["b_in"], c["b_l1"], 24), (c["f1"], c["f2"], c["b_l1"], c["b_l2"], 192)]
    if c["kind"] == "shape":
        return [(c["f0"], c["f1"], c["b0"], c["b1"], 24), (c["f1"], c["f2"], c["b1"], c["b2"], 192),
                (c["f2"], c["f3"], c["b2"], c["b3"], 192)]
    b = c["bandwidth"]
    plan = [(8, 16, b, b // 2), (16, 16, b // 2, b // 2), (16, 24, b // 2, b // 4), (24, 24, b // 4, b // 4),
            (24, 32, b // 4, b // 8), (32, 64, b // 8, b // 8)]
    return [(1, 8, b, b, 6)] + [p + (36,) for p in plan]


def _layer_flops(batch, layer, s2, train, first):
    fi, fo, bi, bo, ng = layer
    analysis = (_s2_flops if s2 else _so3_flops)(batch * fi, bi, bo)
    synthesis = _so3_flops(batch * fo, bo, bo)
    product = 8.0 * batch * fi * fo * (_n3(bo) if s2 else sum((2 * l + 1) ** 3 for l in range(bo)))
    if not train:
        return analysis + synthesis + product
    kernel = 4.0 * fi * fo * ng * (bo * bo if s2 else _n3(bo))
    back = (0 if first else analysis + product)     # the first layer's input wants no gradient
    return analysis + 2 * synthesis + 2 * product + 2 * kernel + back


def work(case):
    c = case
    f = 4.0
    if c["kind"] in ("classify", "deep", "shape"):
        layers, train = _net_layers(c), c["mode"] == "train"
        x = c["batch"] * (layers[0][0] * (2 * layers[0][2]) ** 2)
        nclass = 55 if c["kind"] == "shape" else 10
        params = sum(fi * fo * ng + fo for fi, fo, _, _, ng in layers)
        if c["kind"] == "deep":
            params += 64 * 64 + 64 * 32 + 32 * 10
        else:
            params += layers[-1][1] * nclass
        flops = sum(_layer_flops(c["batch"], l, i == 0, train, i == 0) for i, l in enumerate(layers))
        return {"bytes": f * (x + (2 * params if train else params + c["batch"] * nclass)), "flops": flops}
    if c["kind"] == "layer":
        nx = c["batch"] * c["f_in"] * (2 * c["b_in"]) ** 3
        ny = c["batch"] * c["f_out"] * (2 * c["b_out"]) ** 3
        k = c["f_in"] * c["f_out"] * 192 + c["f_out"]
        lay = (c["f_in"], c["f_out"], c["b_in"], c["b_out"], 192)
        return {"bytes": f * (2 * nx + 2 * ny + 2 * k), "flops": _layer_flops(c["batch"], lay, False, True, False)}
    n = 2 * c["b"]
    if c["kind"] == "so3":
        return {"bytes": f * c["batch"] * (n ** 3 + 2 * _n3(c["b_spec"])), "flops": _so3_flops(c["batch"], c["b"], c["b_spec"])}
    if c["kind"] == "s2":
        return {"bytes": f * c["batch"] * (2 * n * n + 2 * c["b_spec"] ** 2),
                "flops": 2 * _s2_flops(c["batch"], c["b"], c["b_spec"])}
    z = c["batch"] * c["features"]
    mix = 8.0 * z * sum((2 * l + 1) ** 3 for l in range(c["b"]))
    return {"bytes": f * 2 * z * n ** 3, "flops": 2 * _so3_flops(z, c["b"], c["b"]) + mix}


def tolerance(case):
    if case["kind"] in ("so3", "s2", "rotate", "layer"):
        return {"rel": 1e-5}       # float32 sums of up to a few thousand terms
    if case["mode"] == "infer":
        return {"rel": 2e-5}
    # training through ReLUs: an activation within rounding distance of zero may fall on either side,
    # which moves single gradient entries by more than rounding does
    return {"rel": 1e-4, "max": 2e-2}
