"""The calls that a quantization job makes of this framework, as cases to measure.

Every case goes through the public entry points of the package (``gptq_2d``, ``quantizer_int``, ``quantizer_trellis``,
``kron_factors``, ``packed_codes``, ``layer_set``).  ``path`` says which:

``sweep``    ``gptq_2d`` with the affine quantizer, factors and scales in hand: the rounding step of a layer;
``layer``    factor preparation of both Grams, per-row scales and the sweep: one layer from weights and Hessian factors;
``block``    the seven matrices of a decoder block through ``LayerPipeline``: what a layer-set job enqueues;
``factors``  ``feedback_factors_from_grams`` alone: the same Grams serve several bit widths;
``absmax``   ``gptq_2d_super_entry`` with scales taken from the current values of each group of columns;
``trellis``  ``gptq_2d_super_entry`` with a bitshift-trellis code over 16 x 16 super-entries;
``gram``     accumulation of a Hessian factor from calibration activations;
``codes``    rounded matrix to packed integer codes and back.

Inputs.  Weights are Gaussian (sigma 0.02).  The feedback factors of the sweeps have the make-up of a damped Hessian's:
couplings that fall off with the distance of two channels, a few strong far ones per channel, and a weak dense floor, so
near and far feedback both decide codes.  They are mild on purpose: the rounding flow of strongly coupled factors is
chaotic, one value next to a rounding tie changes all that follow, and then no two correct implementations that add in
another order can be compared.  No kernel's work depends on the values.  The ``factors`` inputs are sampled Grams of
heavy-tailed activations with 1 % damping.
"""
import functools
import math
import os
import sys

import torch

PACKAGE = os.path.join(os.getcwd(), "gptq-2d_b200")  # the working folder is the tree that is measured
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import gptq_2d as G  # noqa: E402
import kron_factors as K  # noqa: E402
import layer_set  # noqa: E402
import packed_codes as P  # noqa: E402
import quantizer_int as Q  # noqa: E402
import quantizer_trellis as T  # noqa: E402

DEVICE = "cuda:0"
# (name, m, n) of a decoder block's matrices, in units of the model width (8192 in the full-size layer set)
BLOCK = (("q", 1, 1), ("k", .125, 1), ("v", .125, 1), ("o", 1, 1), ("gate", 3.5, 1), ("up", 3.5, 1), ("down", 1, 3.5))


def listed():
    return [
        # the smallest layer of the test configurations: launches and latency are all there is
        {"name": "sweep 256x256 int4", "path": "sweep", "m": 256, "n": 256, "batch": 0, "dtype": "float32", "bits": 4, "group": 0},
        # odd sizes (a vocabulary remainder, a pruned layer): rows are not whole vectors, the last tiles are ragged
        {"name": "sweep 777x1333 int4", "path": "sweep", "m": 777, "n": 1333, "batch": 0, "dtype": "float32", "bits": 4, "group": 0},
        # a stack of small matrices (experts, heads) under one output-side factor that is broadcast over the stack
        {"name": "sweep 16x512x512 int4", "path": "sweep", "m": 512, "n": 512, "batch": 16, "dtype": "float32", "bits": 4, "group": 0},
        # float64, as a reference run of a small layer uses it
        {"name": "sweep 600x900 int4 float64", "path": "sweep", "m": 600, "n": 900, "batch": 0, "dtype": "float64", "bits": 4, "group": 0},
        # the largest layer: a down projection, scale and zero point per group of 128 columns
        {"name": "sweep 8192x28672 int4 g128", "path": "sweep", "m": 8192, "n": 28672, "batch": 0, "dtype": "float32", "bits": 4, "group": 128},
        # the benchmark's layer: both factors, scales, sweep
        {"name": "layer 8192x8192 int4", "path": "layer", "m": 8192, "n": 8192, "bits": 4},
        # a decoder block of a small model, two layers in flight
        {"name": "block of width 1024", "path": "block", "width": 1024},
        # the factors of the down projection
        {"name": "factors 8192, 28672", "path": "factors", "m": 8192, "n": 28672},
        # INT4 with one scale per group of 32 columns, taken when the group is rounded
        {"name": "absmax 512x2048 groups of 32", "path": "absmax", "m": 512, "n": 2048, "p": 1, "q": 32, "bits": 4},
        # two bits per weight: the HYB code on 256-weight sequences
        {"name": "trellis hyb 512x1024", "path": "trellis", "m": 512, "n": 1024, "code": "hyb", "K": 2},
        # one calibration batch of 8192 tokens into the Hessian factor of 8192 channels
        {"name": "gram 8192 of 8192", "path": "gram", "k": 8192, "n": 8192},
        # storing the result of the largest layer and loading it again
        {"name": "codes 8192x28672 int4", "path": "codes", "m": 8192, "n": 28672, "bits": 4, "group": 0},
    ]


def _size(rng, low, high, step=1):
    """Log-uniform size; every other one is a multiple of 64, the rest whatever it is (in steps of `step`)."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    if rng.random() < .5 and v >= 128:
        step = max(step, 64)
    return max(low, int(round(v / step)) * step)


def draw(rng):
    path = rng.choice(("sweep", "sweep", "sweep", "layer", "block", "factors", "absmax", "trellis", "gram", "codes"))
    if path == "sweep":
        kind = rng.choice(("plain", "plain", "plain", "batch", "float64"))
        top = {"plain": 12288, "batch": 768, "float64": 1200}[kind]
        return {"path": path, "m": _size(rng, 64, top), "n": _size(rng, 64, top), "batch": rng.randint(2, 32) if kind == "batch" else 0,
                "dtype": "float64" if kind == "float64" else "float32", "bits": rng.choice((4, 4, 8)), "group": rng.choice((0, 0, 128))}
    if path == "layer":
        return {"path": path, "m": _size(rng, 128, 8192), "n": _size(rng, 128, 8192), "bits": rng.choice((4, 4, 8))}
    if path == "block":
        return {"path": path, "width": _size(rng, 256, 2048, 16)}
    if path == "factors":
        return {"path": path, "m": _size(rng, 256, 16384), "n": _size(rng, 256, 16384)}
    if path == "absmax":
        q = rng.choice((16, 32, 64, 128))
        return {"path": path, "m": _size(rng, 64, 1024, 4), "n": _size(rng, 256, 4096, q), "p": rng.choice((1, 1, 4)), "q": q, "bits": rng.choice((3, 4, 8))}
    if path == "trellis":
        code = rng.choice(("hyb", "hyb", "one_mad", "three_inst"))
        return {"path": path, "m": _size(rng, 64, 512, 16), "n": _size(rng, 128, 1024, 16), "code": code, "K": rng.choice((2, 2, 3, 4))}
    if path == "gram":
        return {"path": path, "k": _size(rng, 256, 16384), "n": _size(rng, 256, 8192, 4)}
    return {"path": path, "m": _size(rng, 64, 8192), "n": _size(rng, 256, 28672), "bits": rng.choice((2, 3, 4, 4, 8)), "group": rng.choice((0, 0, 128))}


# ---- inputs ----------------------------------------------------------------------------------------------------------

def _couplings(n, generator, dtype, size=1):
    """Strictly lower [n, n] couplings outside the size x size diagonal blocks: falling off over about four (blocks of)
    channels, four far ones per column, and a floor of 0.02 / n."""
    out = torch.empty(n, n, device=DEVICE, dtype=dtype)
    reach = 4.0 * size
    for r0 in range(0, n, 4096):
        r1 = min(n, r0 + 4096)
        part = torch.randn(r1 - r0, n, generator=generator, device=DEVICE, dtype=dtype)
        rows = torch.arange(r0, r1, device=DEVICE, dtype=dtype)[:, None]
        cols = torch.arange(n, device=DEVICE, dtype=dtype)[None, :]
        out[r0:r1] = part * (.05 / size * torch.exp(-(rows - cols).abs() / reach) + .02 / n)
    columns = torch.arange(n, device=DEVICE)[:, None].expand(n, 4)
    far = (columns + 1 + torch.rand(n, 4, generator=generator, device=DEVICE) * (n - 1 - columns)).long().clamp_(max=n - 1)
    sign = torch.randint(0, 2, (n, 4), generator=generator, device=DEVICE).to(dtype) * 2 - 1
    out[far, columns] = .05 / size * sign
    index = torch.arange(n, device=DEVICE) // size
    for r0 in range(0, n, 4096):
        out[r0:r0 + 4096].masked_fill_(index[r0:r0 + 4096, None] <= index[None, :], 0)
    return out


def _factor(n, generator, dtype, size=1):
    """A feedback factor in hand: unit lower triangular, identity diagonal blocks."""
    out = _couplings(n, generator, dtype, size)
    out.diagonal().fill_(1)
    return out


def _gram(n, generator, dtype=torch.float32):
    """A well-conditioned Hessian factor with such couplings and log-normal channel scales (sigma 0.5)."""
    h = _couplings(n, generator, dtype)
    h = h + h.T
    h.diagonal().add_(1)
    d = torch.exp(.5 * torch.randn(n, generator=generator, device=DEVICE, dtype=dtype))
    return h.mul_(d[:, None]).mul_(d[None, :])


def _sampled_gram(n, generator):
    """X^T X / k + 1 % damping for heavy-tailed activations, k = 8192 at most."""
    k = min(8192, 2 * n)
    channel = torch.exp(torch.randn(n, generator=generator, device=DEVICE))
    x = torch.randn(k, n, generator=generator, device=DEVICE) * channel
    h = x.T @ x
    h /= k
    h.diagonal().add_(.01 * h.diagonal().mean())
    return h


def _scales(w, bits, group):
    """The affine quantizer's scale and zero point for w [.., m, n] as a job holds them: one symmetric scale per row
    (broadcast views), or minimum and maximum per group of columns (full matrices)."""
    m, n = w.shape[-2:]
    if not group:
        scale = Q.int_abs_max_scale_cuda(w, qmin=-2 ** (bits - 1), qmax=2 ** (bits - 1) - 1, dtype=torch.float16)
        return scale.expand(w.shape), torch.zeros(1, 1, device=DEVICE, dtype=w.dtype).expand(m, n)
    lo, hi = [], []
    for c in range(0, n, group):
        part = w[..., c:c + group]
        lo.append(part.amin(-1, keepdim=True).expand(part.shape))
        hi.append(part.amax(-1, keepdim=True).expand(part.shape))
    lo, hi = torch.cat(lo, -1), torch.cat(hi, -1)
    scale = (hi - lo).div_(2 ** bits - 1)
    return scale, torch.round(-lo / scale)


def _affine(bits, group):
    low, high = (0, 2 ** bits - 1) if group else (-2 ** (bits - 1), 2 ** (bits - 1) - 1)
    return functools.partial(Q.affine_quantizer_cuda, qmin=low, qmax=high)


def prepare(case, seed):
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    path = case["path"]
    dtype = getattr(torch, case.get("dtype", "float32"))
    weights = lambda *shape: torch.randn(*shape, generator=generator, device=DEVICE, dtype=dtype).mul_(.02)
    if path == "sweep":
        m, n, batch = case["m"], case["n"], case["batch"]
        lead = (batch,) if batch else ()
        w = weights(*lead, m, n)
        l = _factor(m, generator, dtype)
        u = torch.stack([_factor(n, generator, dtype).T.contiguous() for _ in range(batch)]) if batch else _factor(n, generator, dtype).T.contiguous()
        return {"path": path, "w": w, "l": l, "u": u, "inputs": _scales(w, case["bits"], case["group"]), "quantizer": _affine(case["bits"], case["group"])}
    if path == "layer":
        m, n = case["m"], case["n"]
        return {"path": path, "w": weights(m, n), "g": _gram(m, generator), "h": _gram(n, generator), "bits": case["bits"],
                "zero": torch.zeros(1, 1, device=DEVICE).expand(m, n), "quantizer": _affine(case["bits"], 0)}
    if path == "block":
        layers = []
        for _, a, b in BLOCK:
            m, n = int(case["width"] * a), int(case["width"] * b)
            layers.append((weights(m, n), _gram(m, generator), _gram(n, generator)))
        return {"path": path, "layers": layers, "pipeline": layer_set.LayerPipeline(torch.device(DEVICE))}
    if path == "factors":
        return {"path": path, "g": _sampled_gram(case["m"], generator), "h": _sampled_gram(case["n"], generator)}
    if path == "absmax":
        m, n, p, q, bits = (case[k] for k in ("m", "n", "p", "q", "bits"))
        quantizer = functools.partial(Q.int_abs_max_quantizer_cuda, qmin=-2 ** (bits - 1), qmax=2 ** (bits - 1) - 1, dtype=torch.float16)
        return {"path": path, "w": weights(m, n), "l": _factor(m, generator, dtype, p), "u": _factor(n, generator, dtype, q).T.contiguous(),
                "shape": (p, q), "quantizer": quantizer, "inputs": ()}
    if path == "trellis":
        m, n = case["m"], case["n"]
        w = weights(m, n)
        table = getattr(T, case["code"])(L=16, device=DEVICE, dtype=torch.float32)
        scale = w.square().mean().sqrt() / (.9 * table.square().mean().sqrt())
        quantizer = functools.partial(T.trellis_quantizer_super_entry_cuda, table=table, K=case["K"], tail_biting=True)
        return {"path": path, "w": w, "l": _factor(m, generator, dtype, 16), "u": _factor(n, generator, dtype, 16).T.contiguous(),
                "shape": (16, 16), "quantizer": quantizer, "inputs": (scale.reshape(()),)}
    if path == "gram":
        k, n = case["k"], case["n"]
        x = torch.randn(k, n, generator=generator, device=DEVICE) * torch.exp(torch.randn(n, generator=generator, device=DEVICE))
        return {"path": path, "x": x, "h": torch.zeros(n, n, device=DEVICE)}
    m, n, bits, group = case["m"], case["n"], case["bits"], case["group"]
    w = weights(m, n)
    scale, zero = _scales(w, bits, group)
    low, high = (0, 2 ** bits - 1) if group else (-2 ** (bits - 1), 2 ** (bits - 1) - 1)
    z = (torch.clamp(torch.round(w / scale + zero), low, high) - zero) * scale
    return {"path": path, "z": z, "scale": scale, "zero": zero, "qmin": low, "bits": bits}


# ---- one pass --------------------------------------------------------------------------------------------------------

def run(state):
    path = state["path"]
    if path == "sweep":
        return G.gptq_2d(state["w"], state["l"], state["u"], quantizer=state["quantizer"], quantizer_inputs=state["inputs"])
    if path == "layer":
        w, bits = state["w"], state["bits"]
        l, u = K.feedback_factors_from_grams(state["g"], state["h"])
        scale = Q.int_abs_max_scale_cuda(w, qmin=-2 ** (bits - 1), qmax=2 ** (bits - 1) - 1, dtype=torch.float16)
        z = G.gptq_2d(w, l, u, quantizer=state["quantizer"], quantizer_inputs=(scale.expand(w.shape), state["zero"]))
        return {"l": l, "u": u, "scale": scale, "z": z}
    if path == "block":
        return [state["pipeline"].quantize(w, g, h) for w, g, h in state["layers"]]
    if path == "factors":
        return K.feedback_factors_from_grams(state["g"], state["h"])
    if path in ("absmax", "trellis"):
        return G.gptq_2d_super_entry(state["w"], state["l"], state["u"], quantizer=state["quantizer"], super_entry_shape=state["shape"],
                                     quantizer_inputs=state["inputs"])
    if path == "gram":
        return K.accumulate_gram(state["h"].zero_(), state["x"], 1.0 / state["x"].size(0))  # the first batch of a factor
    codes = P.pack_codes(state["z"], state["scale"], state["zero"], qmin=state["qmin"], bits=state["bits"])
    back = P.unpack_codes(codes, state["scale"], state["zero"], qmin=state["qmin"], bits=state["bits"], n=state["z"].size(1))
    return {"codes": codes, "z": back}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------

def _sweep_work(m, n, batch=1, elem=4, group=0, shared_l=1):
    """Weights in and out, one triangle of each factor, the scales as given; two multiply-adds per entry and earlier
    entry of its row and column (half of m + n of them on average)."""
    scales = 2.0 * m * n if group else m
    return {"bytes": elem * (batch * (2.0 * m * n + scales + n * n / 2.0) + shared_l * m * m / 2.0), "flops": float(batch) * m * n * (m + n - 2)}


def _factor_work(n):
    """One triangle in, the full factor out; Cholesky and triangular inverse."""
    return {"bytes": 4.0 * (1.5 * n * n), "flops": 2.0 * n ** 3 / 3}


def _sum(*parts):
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def work(case):
    path = case["path"]
    if path == "sweep":
        return _sweep_work(case["m"], case["n"], max(1, case["batch"]), 8 if case["dtype"] == "float64" else 4, case["group"])
    if path == "layer":
        return _sum(_sweep_work(case["m"], case["n"]), _factor_work(case["m"]), _factor_work(case["n"]))
    if path == "block":
        sizes = [(int(case["width"] * a), int(case["width"] * b)) for _, a, b in BLOCK]
        return _sum(*(w for m, n in sizes for w in (_sweep_work(m, n), _factor_work(m), _factor_work(n))))
    if path == "factors":
        return _sum(_factor_work(case["m"]), _factor_work(case["n"]))
    if path == "absmax":
        return _sweep_work(case["m"], case["n"])
    if path == "trellis":
        # 2^16 states, 256 / V steps, two passes; per state and step 3 V + 1 operations
        values = 2 if case["code"] == "hyb" else 1
        sequences = case["m"] * case["n"] / 256.0
        search = {"bytes": 4.0 * values * 2 ** 16, "flops": sequences * 2 * (3 * values + 1) * 2.0 ** 16 * (256 // values)}
        return _sum(_sweep_work(case["m"], case["n"]), search)
    if path == "gram":
        return {"bytes": 4.0 * (case["k"] * case["n"] + case["n"] ** 2), "flops": float(case["n"]) * (case["n"] + 1) * case["k"]}
    m, n, bits = case["m"], case["n"], case["bits"]
    scales = 2.0 * m * n if case["group"] else m
    return {"bytes": 2 * (4.0 * m * n + m * n * bits / 8.0 + 4.0 * scales), "flops": 0.0}


def tolerance(case):
    """Sums of 32-bit products in another order differ by about 1e-5 of a code at most, so about one value in 1e5 lies close
    enough to a rounding tie to come out one code away, and a few more follow it; one code is up to 1 / 7.5 of the
    largest weight of its row (about half the root mean square).  2-norm: sqrt(8e-5) * 0.55 at most."""
    path = case["path"]
    if path == "codes":
        return "exact"
    if path == "gram":
        return {"rel": 1e-5, "max": 1e-4}
    if path == "factors":
        # damped Grams of condition number 1e4: the inverse factor in 32 bits
        return {"rel": 1e-5, "max": 1e-3}
    if path == "trellis":
        return {"rel": 1e-5, "max": 1e-4}  # the search picks the same path unless its inputs differ
    if case.get("dtype") == "float64":
        return {"rel": 1e-9, "max": 1e-8}
    return {"rel": 5e-3, "max": .99}
