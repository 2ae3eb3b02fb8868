"""Performance cases of the library: the calls its users make, with the sizes they make them at.

`listed()` gives the fixed cases and `draw(rng)` one more from the same ranges.  A case names a
`kind` of call and its sizes; `prepare` builds what a program holds before the call (module, operands,
upstream gradient), `run` makes one call through the public entry points, `work` states the bytes and
operations the call cannot do without and `tolerance` how far another correct implementation of the
same precision may be off.

Units: one (m, n, k) triple of a MAM product is a multiply, a max and a min, three operations; the
backward of one output is four multiply-adds (two selected pairs, two gradients).
"""
import math

import torch

import mamtorch_b200 as mamtorch

# The largest product a drawn case may form, below what the listed ones do.
_MAX_UNITS = 2.0e10


def listed():
    return [
        # A few tokens through the first MLP layer of ViT-B/16 at inference: latency, launches and one read of W.
        {"name": "infer_8_tokens", "kind": "infer", "m": 8, "k": 768, "n": 3072},
        # One optimiser step's forward + backward of a small fully-connected layer: 256 rows, 512 -> 256.
        {"name": "train_small", "kind": "train", "m": 256, "k": 512, "n": 256, "splits": 1},
        # The layer with its reduction cut into slices, second MLP layer of ViT-B/16, 16 images.
        {"name": "train_splits", "kind": "train", "m": 3152, "k": 3072, "n": 768, "splits": 4},
        # The MLP pair of ViT-B/16 as the pruning workflow trains it: 64 images, selection counts on.
        {"name": "vit_mlp_pair", "kind": "mlp", "m": 12608, "k": 768, "n": 3072},
        # The reference-named operator and its backward called directly on sizes that fit no tile.
        {"name": "op_ragged", "kind": "op", "m": 777, "k": 1001, "n": 515},
        # The values-only operator on a large square product.
        {"name": "op_fast_4096", "kind": "fast", "m": 4096, "k": 4096, "n": 4096},
        # A step in the middle of the vanishing-contribution schedule, dense term in TF32.
        {"name": "blend_4096", "kind": "blend", "m": 4096, "k": 4096, "n": 4096, "tf32": True},
        # A convolution layer's training step: a batch of 128 feature maps, 3x3, 64 -> 128 channels.
        {"name": "conv_train", "kind": "conv", "b": 128, "c": 64, "h": 56, "w": 56, "f": 128, "kernel": 3,
         "stride": 1, "order": "unfold"},
        # The same without patch rows, on a strided layer deeper in such a network.
        {"name": "conv_train_taps", "kind": "conv", "b": 32, "c": 128, "h": 28, "w": 28, "f": 256, "kernel": 3,
         "stride": 2, "order": "taps"},
        # Serving a layer pruned to 90 %: a moderate batch on weights that do not change.
        {"name": "pruned_infer", "kind": "pruned_infer", "m": 256, "k": 4096, "n": 4096, "sparsity": 0.9},
        # Fine-tuning the pruned layer: one rank's share of a large batch.
        {"name": "pruned_train", "kind": "pruned_train", "m": 8192, "k": 4096, "n": 4096, "sparsity": 0.9},
        # The ordinary sparse x dense product on the same weight.
        {"name": "spmm_90", "kind": "spmm", "m": 4096, "k": 4096, "n": 4096, "sparsity": 0.9, "layout": "csr"},
    ]


def _size(rng, lo, hi):
    """An extent in [lo, hi], spread over its logarithm: a third each as it comes, on a multiple of 8 and on one
    of 64."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    step = rng.choice((1, 8, 64))
    return int(min(hi, max(lo, round(v / step) * step)))


def _product(rng, m, k, n, most=_MAX_UNITS):
    """Extents from the three (lo, hi) ranges whose product stays within `most`."""
    while True:
        s = _size(rng, *m), _size(rng, *k), _size(rng, *n)
        if s[0] * s[1] * s[2] <= most:
            return dict(zip("mkn", s))


def draw(rng):
    kind = rng.choice(("infer", "train", "mlp", "op", "fast", "blend", "conv", "pruned_infer", "pruned_train", "spmm"))
    case = {"kind": kind}
    if kind == "infer":
        case.update(_product(rng, (1, 4096), (128, 4096), (128, 4096)))
    elif kind == "train":
        case["splits"] = rng.choice((1, 1, 2, 4))
        case.update(_product(rng, (64, 12608), (128, 4096), (64, 4096), 1.5e10))
    elif kind == "mlp":
        width = 32 * rng.randint(6, 32)                # 192 ... 1024, four times as many hidden units
        images = rng.choice((1, 2, 4, 8, 16, 32, 64))
        case.update(m=min(197 * images, int(6e9 // (4 * width * width))), k=width, n=4 * width)
    elif kind == "op":
        case.update(_product(rng, (16, 2048), (16, 2048), (16, 2048), 2e9))
    elif kind == "fast":
        case.update(_product(rng, (64, 4096), (64, 4096), (64, 4096)))
    elif kind == "blend":
        case["tf32"] = rng.random() < 0.5
        case.update(_product(rng, (64, 4096), (64, 4096), (64, 4096), 1e10))
    elif kind == "conv":
        case["kernel"], case["stride"] = rng.choice((1, 3, 3, 5)), rng.choice((1, 1, 2))
        case["order"] = rng.choice(("unfold", "taps"))
        while True:
            b, c, f, side = _size(rng, 1, 128), _size(rng, 3, 256), _size(rng, 16, 256), rng.randint(7, 64)
            units = b * (side // case["stride"] + 1) ** 2 * max(c, 32) * case["kernel"] ** 2 * f
            if units <= 1e10:
                break
        case.update(b=b, c=c, h=side, w=max(7, side + rng.randint(-3, 3)), f=f)
    else:
        case["sparsity"] = round(rng.choice((rng.uniform(0.5, 0.9), rng.uniform(0.9, 0.99))), 3)
        dense = (1.2e10 if kind == "pruned_train" else 6e9) / (1 - case["sparsity"])
        rows = {"pruned_infer": (1, 2048), "pruned_train": (64, 8192), "spmm": (16, 4096)}[kind]
        case.update(_product(rng, rows, (256, 4096), (256, 4096), min(dense, 1.3e11)))
        if kind == "spmm":
            case["layout"] = rng.choice(("csr", "coo"))
    return case


def _normal(gen, *shape, std=1.0):
    return torch.randn(*shape, generator=gen, device="cuda") * std


def _fill(layer, gen, fan_in):
    """Parameters from the seed: N(0, 1/fan_in) weights, small biases."""
    with torch.no_grad():
        layer.weight.copy_(_normal(gen, *layer.weight.shape, std=fan_in ** -0.5))
        if layer.bias is not None:
            layer.bias.copy_(_normal(gen, *layer.bias.shape, std=0.02))
    return layer


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    mamtorch.nn.functional.set_dense_backend("tf32" if case.get("tf32") else "auto")
    s = {"kind": kind}
    if kind == "conv":
        b, c, h, w, f = (case[v] for v in "bchwf")
        r = case["kernel"]
        conv = mamtorch.nn.MAMConv2d(c, f, r, stride=case["stride"], padding=r // 2, reduction_order=case["order"])
        s["layer"] = _fill(conv.cuda(), gen, c * r * r)
        s["x"] = _normal(gen, b, c, h, w).requires_grad_()
        s["gy"] = _normal(gen, b, f, *_out_extent(case))
        return s
    m, k, n = case["m"], case["k"], case["n"]
    if kind == "infer":
        s["layer"] = _fill(mamtorch.nn.FullyConnected(k, n, device="cuda"), gen, k).eval()
        s["x"] = _normal(gen, m, k)
    elif kind == "train":
        s["layer"] = _fill(mamtorch.nn.FullyConnected(k, n, splits=case["splits"], device="cuda"), gen, k)
        s["x"] = _normal(gen, m, k).requires_grad_()
        s["gy"] = _normal(gen, m, n)
    elif kind == "mlp":
        s["fc1"] = _fill(mamtorch.nn.FullyConnected(k, n, store_args=True, device="cuda"), gen, k)
        s["fc2"] = _fill(mamtorch.nn.FullyConnected(n, k, store_args=True, device="cuda"), gen, n)
        s["x"] = _normal(gen, m, k).requires_grad_()
        s["gy"] = _normal(gen, m, k)
    elif kind == "op":
        # activations as a ReLU leaves them
        s["a"] = _normal(gen, m, k).relu_().requires_grad_()
        s["b"] = _normal(gen, k, n, std=k ** -0.5).requires_grad_()
        s["gy"] = _normal(gen, m, n)
    elif kind == "fast":
        s["a"], s["b"] = _normal(gen, m, k), _normal(gen, k, n, std=k ** -0.5)
    elif kind == "blend":
        s["layer"] = _fill(mamtorch.nn.FullyConnected(k, n, vcon_steps=2, device="cuda"), gen, k)
        s["layer"].vcon_step()                         # beta 1 -> 0.5
        s["x"] = _normal(gen, m, k).requires_grad_()
        s["gy"] = _normal(gen, m, n)
    elif kind in ("pruned_infer", "pruned_train"):
        dense = _fill(mamtorch.nn.FullyConnected(k, n, device="cuda"), gen, k)
        s["layer"] = mamtorch.sparse.PrunedFullyConnected.from_dense(dense, fraction=case["sparsity"])
        s["x"] = _normal(gen, m, k)
        if kind == "pruned_train":
            s["x"].requires_grad_()
            s["gy"] = _normal(gen, m, n)
    else:
        # the sparse operand is the weight [n, k], the dense one holds m columns
        keep = torch.rand(n, k, generator=gen, device="cuda") >= case["sparsity"]
        keep[0, 0] = True
        w = _normal(gen, n, k) * keep
        s["a"] = w.to_sparse_csr() if case["layout"] == "csr" else w.to_sparse_coo().coalesce()
        s["b"] = _normal(gen, k, m)
    return s


def _step(s, layer):
    """Forward + backward of one layer, gradients fresh as after optimizer.zero_grad()."""
    s["x"].grad = layer.weight.grad = layer.bias.grad = None
    y = layer(s["x"])
    y.backward(s["gy"])
    return {"y": y.detach(), "dx": s["x"].grad, "dw": layer.weight.grad, "db": layer.bias.grad}


def run(s):
    kind = s["kind"]
    if kind == "infer":
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind in ("train", "blend"):
        return _step(s, s["layer"])
    if kind == "conv":
        out = _step(s, s["layer"])
        out.update(argmax=s["layer"].argmax, argmin=s["layer"].argmin)
        return out
    if kind == "mlp":
        fc1, fc2, x = s["fc1"], s["fc2"], s["x"]
        params = (fc1.weight, fc1.bias, fc2.weight, fc2.bias)
        for t in (x, *params):
            t.grad = None
        y = fc2(fc1(x))
        y.backward(s["gy"])
        fc1.update_selection_count()
        fc2.update_selection_count()
        return [y.detach(), x.grad, *(p.grad for p in params), fc1.max_selection_count, fc2.max_selection_count]
    if kind == "op":
        a, b = s["a"], s["b"]
        a.grad = b.grad = None
        y, argmax, argmin = mamtorch.kernel.v4.fullyconnected(a, b)
        y.backward(s["gy"])
        return [y.detach(), argmax, argmin, a.grad, b.grad]
    if kind == "fast":
        return mamtorch.kernel.v4.fullyconnected_fast(s["a"], s["b"])
    if kind == "pruned_infer":
        with torch.no_grad():
            y = s["layer"](s["x"])
        return [y, s["layer"].argmax, s["layer"].argmin]
    if kind == "pruned_train":
        out = _step(s, s["layer"])
        out.update(argmax=s["layer"].argmax, argmin=s["layer"].argmin)
        return out
    return mamtorch.sparse.kernel.v1.cusparsemm(s["a"], s["b"])


def _out_extent(case):
    r, st = case["kernel"], case["stride"]
    return tuple((case[v] + 2 * (r // 2) - r) // st + 1 for v in "hw")


def work(case):
    kind = case["kind"]
    if kind == "conv":
        ho, wo = _out_extent(case)
        m, k, n = case["b"] * ho * wo, case["c"] * case["kernel"] ** 2, case["f"]
        x_size = case["b"] * case["c"] * case["h"] * case["w"]
        # x, w, gy in; y, two index matrices, dx, dw out
        return {"bytes": 4 * (2 * x_size + 2 * n * k + 4 * m * n + 2 * n), "flops": 3 * m * n * k + 8 * m * n}
    m, k, n = case["m"], case["k"], case["n"]
    if kind in ("infer", "fast"):
        return {"bytes": 4 * (m * k + n * k + m * n), "flops": 3 * m * n * k}
    if kind == "train":
        return {"bytes": 4 * (2 * m * k + 2 * n * k + 2 * m * n + 2 * n),
                "flops": 3 * m * n * k + 8 * m * n * case["splits"]}
    if kind == "mlp":
        # x, gy, y, dx; both weights, their gradients and counts (read and written)
        return {"bytes": 4 * (4 * m * k + 8 * n * k + 2 * (n + k)), "flops": 6 * m * n * k + 8 * m * (n + k)}
    if kind == "op":
        return {"bytes": 4 * (2 * m * k + 2 * n * k + 4 * m * n), "flops": 3 * m * n * k + 8 * m * n}
    if kind == "blend":
        # the MAM product and three dense ones (forward, two gradients)
        return {"bytes": 4 * (2 * m * k + 2 * n * k + 2 * m * n + 2 * n), "flops": 9 * m * n * k + 8 * m * n}
    nnz = n * k * (1 - case["sparsity"])
    if kind == "pruned_infer":
        return {"bytes": 4 * (m * k + 3 * m * n) + 8 * nnz, "flops": 3 * m * nnz}
    if kind == "pruned_train":
        # the gradient is the dense parameter's
        return {"bytes": 4 * (2 * m * k + 4 * m * n + 2 * n * k) + 8 * nnz, "flops": 3 * m * nnz + 8 * m * n}
    return {"bytes": 4 * (k * m + n * m) + 8 * nnz, "flops": 2 * m * nnz}


def tolerance(case):
    kind = case["kind"]
    if kind in ("infer", "fast", "pruned_infer"):
        return "exact"       # one rounded product each for max and min, one addition: no freedom in the order
    if case.get("tf32"):
        return {"rel": 1e-3}   # 11 significant bits in the dense products
    return {"rel": 1e-5}     # fp32 sums in any order; indices and counts stay whole numbers and the same
