"""The work that programs give this library, for timing and for comparing results.

Each case is a call or a short sequence of calls of the package's public functions, on the kind
of tensors those calls meet in use: the gates of a recurrent cell, a vector times a weight
matrix, the products of an MLP training step, of an attention block and of conv layers (forward
and backward), single products from small to large, ragged ones, float64, integers, and products
on host arrays.  ``listed()`` gives one or two cases of each kind, ``draw()`` more of the same
ranges.
"""
import math

import numpy as np
import torch

import tinytensor_b200 as ttb

DTYPES = {"f32": torch.float32, "f64": torch.float64, "u8": torch.uint8, "i16": torch.int16, "i32": torch.int32,
          "i64": torch.int64}
SIZE = {"f32": 4, "f64": 8, "u8": 1, "i16": 2, "i32": 4, "i64": 8}


def listed():
    return [
        # Gates of an LSTM cell at one time step, the smallest calls there are: x.Wx + b, then h.Wh added to it.
        {"name": "cell_32x128", "kind": "cell", "n": 32, "inputs": 64, "hidden": 128},
        # One token / one sample through a weight matrix: vector times matrix, nothing but reading the weights.
        {"name": "vecmat_4096", "kind": "vecmat", "k": 4096, "m": 4096},
        # An everyday square product.
        {"name": "matmul_512", "kind": "matmul", "n": 512, "k": 512, "m": 512},
        # Large enough that only the arithmetic rate counts.
        {"name": "matmul_8192", "kind": "matmul", "n": 8192, "k": 8192, "m": 8192},
        # MNIST classifier 784 -> 1024 -> 10, batch 4096: both layers forward, both layers backward.
        {"name": "mlp_4096", "kind": "mlp", "n": 4096, "inputs": 784, "hidden": 1024, "classes": 10},
        # Attention products of 256 heads of 128 tokens x 64 channels, forward and backward.
        {"name": "attention_256x128x64", "kind": "attention", "b": 256, "t": 128, "d": 64},
        # Forward and backward of a product none of whose sizes is a multiple of anything useful.
        {"name": "train_ragged", "kind": "train", "dtype": "f32", "b": 1, "n": 1003, "k": 769, "m": 1251},
        # Forward and backward in double precision.
        {"name": "train_f64", "kind": "train", "dtype": "f64", "b": 1, "n": 2048, "k": 1024, "m": 1536},
        # Batched product of small whole numbers (one-hot and count data, quantised values).
        {"name": "int_i32_64x1024", "kind": "int", "dtype": "i32", "b": 64, "n": 1024, "k": 512, "m": 1024, "most": 8},
        # A middle layer of an image network, forward and backward.
        {"name": "conv_64_128_56", "kind": "conv", "b": 32, "c_in": 64, "hw": 56, "c_out": 128, "kernel": 3, "stride": 1,
         "padding": 1},
        # The first layer of a digit classifier, forward and backward.
        {"name": "conv_1_32_28", "kind": "conv", "b": 64, "c_in": 1, "hw": 28, "c_out": 32, "kernel": 5, "stride": 1,
         "padding": 0},
        # A caller whose arrays are numpy arrays in ordinary memory.
        {"name": "host_1024", "kind": "host", "b": 1, "n": 1024, "k": 1024, "m": 1024},
    ]


def _size(rng, low, high):
    """A size, spread over the logarithm of the range; every other one is a multiple of 8 where that fits."""
    v = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    if v >= 16 and rng.random() < 0.5:
        v = (v + 4) // 8 * 8
    return max(low, min(high, v))


def draw(rng):
    kind = rng.choice(["cell", "vecmat", "matmul", "mlp", "attention", "train", "train64", "int", "conv", "host"])
    if kind == "cell":
        return {"kind": "cell", "n": _size(rng, 1, 256), "inputs": _size(rng, 8, 512), "hidden": _size(rng, 8, 256)}
    if kind == "vecmat":
        return {"kind": "vecmat", "k": _size(rng, 64, 8192), "m": _size(rng, 64, 8192)}
    if kind == "matmul":
        return {"kind": "matmul", "n": _size(rng, 16, 8192), "k": _size(rng, 16, 8192), "m": _size(rng, 16, 8192)}
    if kind == "mlp":
        return {"kind": "mlp", "n": _size(rng, 32, 8192), "inputs": _size(rng, 32, 2048), "hidden": _size(rng, 32, 2048),
                "classes": _size(rng, 2, 128)}
    if kind == "attention":
        t = _size(rng, 16, 512)
        return {"kind": "attention", "b": _size(rng, 4, max(8, min(512, (1 << 24) // (t * t)))), "t": t,
                "d": _size(rng, 16, 128)}
    if kind == "train":
        return {"kind": "train", "dtype": "f32", "b": rng.choice([1, 1, 2, 8]), "n": _size(rng, 64, 2048),
                "k": _size(rng, 64, 2048), "m": _size(rng, 64, 2048)}
    if kind == "train64":
        return {"kind": "train", "dtype": "f64", "b": rng.choice([1, 1, 4]), "n": _size(rng, 32, 2048),
                "k": _size(rng, 32, 1024), "m": _size(rng, 32, 1536)}
    if kind == "int":
        dtype = rng.choice(["i32", "i32", "i64", "i16", "u8"])
        return {"kind": "int", "dtype": dtype, "b": _size(rng, 1, 8 if dtype == "i64" else 64),
                "n": _size(rng, 16, 1024), "k": _size(rng, 16, 512), "m": _size(rng, 16, 1024),
                "most": rng.choice([8, 100, 30000, 2000000000])}
    if kind == "conv":
        kernel = rng.choice([1, 3, 3, 3, 5])
        hw = _size(rng, max(7, kernel), 64)
        c_in = rng.choice([1, 3, _size(rng, 8, 128), _size(rng, 8, 128)])
        return {"kind": "conv", "b": _size(rng, 1, 32), "c_in": c_in, "hw": hw, "c_out": _size(rng, 8, 128),
                "kernel": kernel, "stride": rng.choice([1, 1, 2]), "padding": rng.choice([0, kernel // 2])}
    return {"kind": "host", "b": rng.choice([1, 1, 4]), "n": _size(rng, 32, 1024), "k": _size(rng, 32, 1024),
            "m": _size(rng, 32, 1024)}


def _out_hw(case):
    return (case["hw"] + 2 * case["padding"] - case["kernel"]) // case["stride"] + 1


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host":
        rng = np.random.default_rng(seed)
        shape_a, shape_b = (case["b"], case["n"], case["k"]), (case["b"], case["k"], case["m"])
        return {"kind": kind, "a": rng.standard_normal(shape_a, dtype=np.float32),
                "b": rng.standard_normal(shape_b, dtype=np.float32)}
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0, dtype=torch.float32):
        return torch.randn(shape, generator=g, device="cuda", dtype=dtype) * std

    s = {"kind": kind}
    if kind == "cell":
        n, i, h = case["n"], case["inputs"], case["hidden"]
        s.update(x=normal(n, i), h=normal(1, n, h, std=0.5), wx=normal(i, 4 * h, std=i ** -0.5),
                 wh=normal(1, h, 4 * h, std=h ** -0.5), bias=normal(4 * h, std=0.1))
    elif kind == "vecmat":
        s.update(a=normal(case["k"]), b=normal(case["k"], case["m"], std=case["k"] ** -0.5))
    elif kind == "matmul":
        s.update(a=normal(case["n"], case["k"]), b=normal(case["k"], case["m"], std=case["k"] ** -0.5))
    elif kind == "mlp":
        n, i, h, c = case["n"], case["inputs"], case["hidden"], case["classes"]
        s.update(x=torch.rand((n, i), generator=g, device="cuda"), w1=normal(i, h, std=i ** -0.5), b1=normal(h, std=0.1),
                 w2=normal(h, c, std=h ** -0.5), b2=normal(c, std=0.1), dy=normal(n, c, std=1.0 / n))
    elif kind == "attention":
        b, t, d = case["b"], case["t"], case["d"]
        s.update(q=normal(b, t, d, std=d ** -0.5), k=normal(b, t, d), v=normal(b, t, d), g=normal(b, t, d))
    elif kind == "train":
        b, n, k, m, dt = case["b"], case["n"], case["k"], case["m"], DTYPES[case["dtype"]]
        lead = (b,) if b > 1 else ()
        s.update(a=normal(*lead, n, k, dtype=dt), b=normal(*lead, k, m, std=k ** -0.5, dtype=dt),
                 g=normal(*lead, n, m, dtype=dt))
    elif kind == "int":
        dt = DTYPES[case["dtype"]]
        info = torch.iinfo(dt)
        low, high = max(info.min, -case["most"]), min(info.max, case["most"]) + 1
        for key, shape in (("a", (case["b"], case["n"], case["k"])), ("b", (case["b"], case["k"], case["m"]))):
            s[key] = torch.randint(low, high, shape, generator=g, device="cuda", dtype=dt)
    else:
        b, ci, hw, co, ks = case["b"], case["c_in"], case["hw"], case["c_out"], case["kernel"]
        ho = _out_hw(case)
        s.update(x=normal(b, ci, hw, hw), w=normal(co, ci, ks, ks, std=(ci * ks * ks) ** -0.5), bias=normal(co, std=0.1),
                 g=normal(b, co, ho, ho), stride=case["stride"], padding=case["padding"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "cell":
        gates = ttb.linear(s["x"], s["wx"], s["bias"])
        return ttb.batched_matmul_fused(s["h"], s["wh"], gates)
    if kind in ("vecmat", "matmul", "int"):
        return ttb.matmul(s["a"], s["b"])
    if kind == "mlp":
        h = ttb.linear(s["x"], s["w1"], s["b1"], ttb.Activation.RELU)
        y = ttb.linear(h, s["w2"], s["b2"])
        dh, dw2 = ttb.matmul_backward(h, s["w2"], s["dy"])
        dx, dw1 = ttb.matmul_backward(s["x"], s["w1"], dh)
        return [h, y, dh, dw2, dx, dw1]
    if kind == "attention":
        kt = s["k"].permute(0, 2, 1)
        p = ttb.matmul(s["q"], kt)
        o = ttb.matmul(p, s["v"])
        dp, dv = ttb.matmul_backward(p, s["v"], s["g"])
        dq, dkt = ttb.matmul_backward(s["q"], kt, dp)
        return [p, o, dp, dv, dq, dkt]
    if kind == "train":
        c = ttb.matmul(s["a"], s["b"])
        da, db = ttb.matmul_backward(s["a"], s["b"], s["g"])
        return [c, da, db]
    if kind == "conv":
        y = ttb.conv2d(s["x"], s["w"], s["bias"], s["stride"], s["padding"])
        gx, gw, gb = ttb.conv2d_backward(s["g"], s["x"], s["w"], s["stride"], s["padding"])
        return [y, gx, gw, gb]
    return ttb.batched_matmul_host(s["a"], s["b"])


def work(case):
    """Bytes and operations of one pass: each input read once, each output written once, 2 n k m a product."""
    kind = case["kind"]
    if kind == "cell":
        n, i, h4 = case["n"], case["inputs"], 4 * case["hidden"]
        h = case["hidden"]
        return {"bytes": 4 * (n * i + n * h + (i + h) * h4 + h4 + n * h4), "flops": 2 * n * (i + h) * h4}
    if kind == "vecmat":
        return {"bytes": 4 * (case["k"] + case["k"] * case["m"] + case["m"]), "flops": 2 * case["k"] * case["m"]}
    if kind == "mlp":
        n, i, h, c = case["n"], case["inputs"], case["hidden"], case["classes"]
        return {"bytes": 4 * (2 * n * i + 2 * i * h + h + 2 * n * h + 2 * h * c + c + 2 * n * c),
                "flops": 6 * n * (i * h + h * c)}
    if kind == "attention":
        b, t, d = case["b"], case["t"], case["d"]
        return {"bytes": 4 * b * (8 * t * d + 2 * t * t), "flops": 12 * b * t * t * d}
    if kind == "conv":
        hw, ho = case["hw"] ** 2, _out_hw(case) ** 2
        b, ci, co, ckk = case["b"], case["c_in"], case["c_out"], case["c_in"] * case["kernel"] ** 2
        return {"bytes": 4 * (2 * b * ci * hw + 2 * b * co * ho + 2 * co * ckk + 2 * co), "flops": 6 * b * co * ckk * ho}
    b, n, k, m = case.get("b", 1), case["n"], case["k"], case["m"]
    if kind == "train":
        return {"bytes": 2 * SIZE[case["dtype"]] * b * (n * k + k * m + n * m), "flops": 6 * b * n * k * m}
    return {"bytes": SIZE[case.get("dtype", "f32")] * b * (n * k + k * m + n * m), "flops": 2 * b * n * k * m}


def tolerance(case):
    if case["kind"] == "int":
        return "exact"  # sums wrap modulo 2^width: every correct implementation gives the same
    if case.get("dtype") == "f64":
        return {"rel": 1e-14, "max": 1e-12}
    return {"rel": 1e-5, "max": 1e-4}
