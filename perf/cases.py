"""Cases of the quantized-linear path: what a program that serves a transformer with this package calls.

A case is a dict of plain values.  ``kind`` names the call chain, through public entry points only:

* ``linear``     a module layer (``NVFP4Linear`` / ``MXFP8Linear``) on a dense activation
* ``layout``     ``QuantizedTensor.from_float(x)`` and ``F.linear`` on two quantized tensors
* ``operators``  ``ck.quantize_*`` of the activation, then ``ck.scaled_mm_*``
* ``gemm``       ``ck.scaled_mm_*`` on operands that are quantized already
* ``mlp``        ``NVFP4MLP`` with a static hidden scale (fc1, GELU, re-quantize, fc2)
* ``quantize``   ``QuantizedTensor.from_float`` of a tensor (weights of a checkpoint)
* ``dequantize`` ``QuantizedTensor.dequantize`` (weights of a layer that needs them dense)

``m`` counts tokens, ``k`` input and ``n`` output features (``mlp``: ``n`` hidden features).  Sizes
are those of the MMDiT-shaped stack and of the benchmark: hidden 3072, MLP 12288, 512 text and 4096
image tokens, batch up to 8.
"""
from __future__ import annotations

import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "comfy-kitchen_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import comfy_kitchen as ck  # noqa: E402
from comfy_kitchen.modules import MXFP8Linear, NVFP4Linear, NVFP4MLP  # noqa: E402
from comfy_kitchen.tensor import QuantizedTensor  # noqa: E402

LAYOUT = {"nvfp4": "TensorCoreNVFP4Layout", "mxfp8": "TensorCoreMXFP8Layout"}
DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
ELEMENT = {"bf16": 2, "fp16": 2, "fp32": 4}
LARGEST = 36864 * 9216 * 3072  # multiply-adds of the largest listed case


def _case(kind, layout, m, n, k, dtype="bf16", bias=True, static=False, **name):
    return {**name, "kind": kind, "layout": layout, "m": m, "n": n, "k": k, "dtype": dtype, "bias": bias, "static": static}


def listed():
    return [
        # modulation vectors of a batch of 8: one row per sample, six chunks of the hidden size
        _case("linear", "nvfp4", 8, 18432, 3072, name="modulation_8_rows"),
        # a single token through the second projection of an MLP
        _case("linear", "mxfp8", 1, 3072, 12288, bias=False, name="one_token_long_k"),
        # pre-quantized operands, few rows and a long K, full-precision result
        _case("gemm", "nvfp4", 256, 3072, 12288, dtype="fp32", bias=False, static=True, name="gemm_256_rows_long_k"),
        # the text stream of one sample, calibrated activation scale, half precision
        _case("linear", "nvfp4", 512, 3072, 3072, dtype="fp16", static=True, name="text_tokens"),
        # a ragged token count through the tensor subclass (rows are padded to the block size)
        _case("layout", "nvfp4", 1003, 9216, 3072, name="ragged_tokens_subclass"),
        # one image-token projection by operators: the benchmark's default step
        _case("operators", "nvfp4", 4096, 3072, 3072, static=True, name="projection_operators"),
        # the same projection in the other format through its module
        _case("linear", "mxfp8", 4096, 3072, 3072, name="projection_mxfp8"),
        # the MLP pair over image and text tokens of one sample
        _case("mlp", "nvfp4", 4608, 12288, 3072, static=True, name="mlp_pair"),
        # second MLP projection of a batch of 4, no bias
        _case("linear", "mxfp8", 16384, 3072, 12288, bias=False, name="batch_long_k_mxfp8"),
        # query/key/value projection of a batch of 8, dynamic activation scale
        _case("linear", "nvfp4", 36864, 9216, 3072, name="batch_qkv"),
        # a checkpoint's MLP weight, stored in fp32, quantized on load
        _case("quantize", "nvfp4", 12288, 0, 3072, dtype="fp32", bias=False, name="quantize_weight_fp32"),
        # the same weight back to dense, for a caller outside the tensor-core path
        _case("dequantize", "nvfp4", 12288, 0, 3072, bias=False, name="dequantize_weight"),
    ]


def _spread(rng, lo, hi, step):
    """A multiple of ``step`` in [lo, hi], uniform over the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi, max(lo, int(round(v / step)) * step or step))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["layout"] * 2 + ["operators"] * 2 + ["gemm", "mlp", "quantize", "dequantize"])
    layout = "nvfp4" if kind == "mlp" else rng.choice(["nvfp4", "nvfp4", "mxfp8"])
    # feature counts: usually multiples of 64, now and then the smallest granule the format takes
    k = _spread(rng, 1024, 15360, rng.choice([64, 64, 64, 32]))
    n = _spread(rng, 1024, 18432, 64 if kind == "mlp" else rng.choice([64, 64, 64, 32 if layout == "mxfp8" else 16]))
    m = _spread(rng, 1, 36864, 1)
    if rng.random() < 0.5 and m > 64:
        m -= m % 64
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
    if kind == "mlp":
        k, n = min(k, 6144), min(max(n, k), 15360)
        dtype = rng.choice(["bf16", "fp16"])
        m = min(m, LARGEST // (2 * n * k))
    if kind in ("quantize", "dequantize"):
        m, n = max(m, 256), 0
    else:
        m = min(m, LARGEST // (n * k))
        if kind == "operators":  # the operators take rows as they are
            m = max(1, m - m % 16) if m > 16 else m
    return _case(kind, layout, max(1, m), n, k, dtype=dtype, bias=n > 0 and rng.random() < 0.7,
                 static=layout == "nvfp4" and (kind in ("operators", "gemm", "mlp") or rng.random() < 0.4))


# ------------------------------------------------------------------------------------------ state
def _activation(gen, m, k, dtype):
    """N(0, 1) with one entry in a thousand scaled by 20, as the projections of a transformer see."""
    x = torch.empty(m, k, dtype=dtype, device="cuda")
    for r in range(0, m, 4096):
        part = torch.randn(min(4096, m - r), k, generator=gen, device="cuda")
        hot = torch.rand(part.shape, generator=gen, device="cuda") < 0.001
        x[r:r + part.shape[0]] = torch.where(hot, part * 20, part)
    return x


def _weight(gen, n, k, dtype):
    return (torch.randn(n, k, generator=gen, device="cuda") * 0.02).to(dtype)


def _dense_linear(gen, n, k, dtype, bias):
    lin = torch.nn.Linear(k, n, bias=bias, device="cuda", dtype=dtype)
    with torch.no_grad():
        lin.weight.copy_(_weight(gen, n, k, dtype))
        if bias:
            lin.bias.copy_(torch.randn(n, generator=gen, device="cuda") * 0.01)
    return lin


def _scale(x):
    return (x.abs().amax() / 2688.0).to(torch.float32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, layout, dtype = case["kind"], case["layout"], DTYPE[case["dtype"]]
    m, n, k, with_bias = case["m"], case["n"], case["k"], case["bias"]
    name = LAYOUT[layout]
    s = {"kind": kind, "layout": layout, "dtype": dtype, "name": name, "scale": None}
    with torch.inference_mode():
        if kind == "quantize":
            s["x"] = _weight(gen, m, k, dtype)
            s["scale"] = _scale(s["x"]) if case["static"] else None
            return s
        if kind == "dequantize":
            s["w"] = QuantizedTensor.from_float(_weight(gen, m, k, dtype), name)
            return s
        x = _activation(gen, m, k, dtype)
        if kind == "mlp":
            fc1 = NVFP4Linear.from_linear(_dense_linear(gen, n, k, dtype, with_bias), input_scale=_scale(x))
            fc2 = NVFP4Linear.from_linear(_dense_linear(gen, k, n, dtype, with_bias))
            s["layer"] = NVFP4MLP(fc1, fc2)
            s["layer"].calibrate(x[:1024])
            s["x"] = x
            return s
        lin = _dense_linear(gen, n, k, dtype, with_bias)
        if kind == "linear":
            if layout == "nvfp4":
                s["layer"] = NVFP4Linear.from_linear(lin, input_scale=_scale(x) if case["static"] else None)
            else:
                s["layer"] = MXFP8Linear.from_linear(lin)
            s["x"] = x
            return s
        s["w"] = QuantizedTensor.from_float(lin.weight.detach(), name)
        s["bias"] = lin.bias.detach() if with_bias else None
        if kind == "gemm":
            s["x"] = QuantizedTensor.from_float(x, name)
        else:
            s["x"] = x
            if layout == "nvfp4" and case["static"]:
                s["scale"] = _scale(x)
        return s


# ------------------------------------------------------------------------------------------ one pass
def _scaled_mm(s, codes, scale, block_scale):
    w, bias, dtype = s["w"], s["bias"], s["dtype"]
    if s["layout"] == "nvfp4":
        return ck.scaled_mm_nvfp4(codes, w._qdata, scale, w.params.scale, block_scale, w.params.block_scale, bias=bias,
                                  out_dtype=dtype)
    return ck.scaled_mm_mxfp8(codes, w._qdata, block_scale, w.params.scale, bias=bias, out_dtype=dtype)


def run(s):
    kind = s["kind"]
    with torch.inference_mode():
        if kind in ("linear", "mlp"):
            return s["layer"](s["x"])
        if kind == "layout":
            xq = QuantizedTensor.from_float(s["x"], s["name"], scale=s["scale"])
            return torch.nn.functional.linear(xq, s["w"], s["bias"])
        if kind == "operators":
            if s["layout"] == "nvfp4":
                codes, block_scale = ck.quantize_nvfp4(s["x"], s["scale"])
            else:
                codes, block_scale = ck.quantize_mxfp8(s["x"])
            return _scaled_mm(s, codes, s["scale"], block_scale)
        if kind == "gemm":
            x = s["x"]
            if s["layout"] == "nvfp4":
                return _scaled_mm(s, x._qdata, x.params.scale, x.params.block_scale)
            return _scaled_mm(s, x._qdata, None, x.params.scale)
        if kind == "quantize":
            q = QuantizedTensor.from_float(s["x"], s["name"], scale=s["scale"])
            if s["layout"] == "nvfp4":
                return q._qdata, q.params.block_scale.view(torch.uint8), q.params.scale
            return q._qdata.view(torch.uint8), q.params.scale.view(torch.uint8)
        return s["w"].dequantize()


# ------------------------------------------------------------------------------------------ what it takes
def work(case):
    m, n, k = case["m"], case["n"], case["k"]
    dense = ELEMENT[case["dtype"]]
    quantized = 0.5 + 1 / 16 if case["layout"] == "nvfp4" else 1 + 1 / 32  # bytes of an element with its block scale
    kind = case["kind"]
    if kind in ("quantize", "dequantize"):
        return {"bytes": m * k * (dense + quantized), "flops": 0}
    if kind == "mlp":
        return {"bytes": 2 * m * k * dense + 2 * n * k * quantized, "flops": 4 * m * n * k}
    return {"bytes": m * k * (quantized if kind == "gemm" else dense) + n * k * quantized + m * n * dense, "flops": 2 * m * n * k}


def tolerance(case):
    """Four times what the path shows against the same chain in 64 bits (same codes and scales).

    Rounding of the result to 16 bits is what moves: up to 4e-4 of the values of a bf16 result lie on
    the other side of a rounding boundary (3.8e-4 in the 2-norm for one row, where one such value
    already counts).  fp16: below 7e-6, or one value of a short row (1.5e-5).  fp32: below 8e-7.
    The MLP's hidden tensor is re-quantized: 1.5e-4 of its values one bf16 step away move about
    2e-6 of the codes by one, which is 5e-4 of the result beside its own rounding.
    """
    if case["kind"] in ("quantize", "dequantize"):
        return "exact"  # codes, scales and decoded values are defined bit for bit
    if case["kind"] == "mlp":
        return {"rel": 4e-3}
    return {"rel": {"bf16": 1.6e-3, "fp16": 1e-4, "fp32": 4e-6}[case["dtype"]]}


# ------------------------------------------------------------------------------------------ in 64 bits
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
_E2M1_MIDDLE = (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0)  # a tie goes to the even code: up behind the odd ones


def _divided(a, b):
    """a / b in fp32, rounded once (a Python number as the divisor would become a product)."""
    return a / torch.as_tensor(b, dtype=torch.float32, device=a.device).expand_as(a)


def _tiled(scales):
    """Scale bytes [rows, columns] in the 128 x 4 tiles that the tensor cores read, zero padded."""
    rows, cols = scales.shape
    r, c = (rows + 127) // 128, (cols + 3) // 4
    full = torch.zeros(r * 128, c * 4, dtype=torch.uint8, device=scales.device)
    full[:rows, :cols] = scales
    return full.view(r, 4, 32, c, 4).permute(0, 3, 2, 1, 4).reshape(r * 128, c * 4)


def _dynamic_scale(x):
    """amax / (448 * 6), divided in x's own type."""
    return _divided(x.abs().amax().float(), 2688.0).to(x.dtype).float()


def _nvfp4(x, scale):
    """(codes 0..15 as uint8, E4M3 scales of 16 elements) of a part of x's rows."""
    v = x.float().view(x.shape[0], -1, 16)
    amax = v.abs().amax(-1)
    block = _divided(_divided(amax, 6.0), scale).clamp(max=448.0).to(torch.float8_e4m3fn)
    total = (scale * block.float()).unsqueeze(-1)
    q = torch.where(total == 0, torch.zeros_like(v), v / torch.where(total == 0, 1.0, total).expand_as(v))
    a = q.abs()
    code = torch.zeros(a.shape, dtype=torch.uint8, device=x.device)
    for i, middle in enumerate(_E2M1_MIDDLE):
        code += (a >= middle) if i % 2 else (a > middle)
    return (code | (torch.signbit(q).to(torch.uint8) << 3)).view(x.shape), block


def _mxfp8(x):
    """(E4M3 data, E8M0 scale bytes of 32 elements) of a part of x's rows."""
    v = x.float().view(x.shape[0], -1, 32)
    amax = v.abs().amax(-1)
    mantissa, exponent = torch.frexp(_divided(amax, 448.0).clamp(min=2.0 ** -127))
    e = (exponent - (mantissa == 0.5).to(exponent.dtype) + 127).clamp(0, 254)
    data = torch.ldexp(v, (127 - e).unsqueeze(-1)).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return data.view(x.shape), torch.where(amax == 0, 0, e).to(torch.uint8)


def _stored(x, layout, scale=None):
    """What the quantized x stands for, in 64 bits."""
    out = torch.empty(x.shape, dtype=torch.float64, device=x.device)
    lut = torch.tensor(_E2M1, dtype=torch.float64, device=x.device)
    for r in range(0, x.shape[0], 2048):
        part = x[r:r + 2048]
        if layout == "nvfp4":
            code, block = _nvfp4(part, scale)
            value = lut[(code & 7).long()] * (1.0 - 2.0 * (code >> 3).double())
            factor, size = block.double() * scale.double(), 16
        else:
            data, e = _mxfp8(part)
            value, size = data.double(), 32
            factor = torch.where(e == 0, 0.0, torch.ldexp(torch.ones_like(e, dtype=torch.float64), e.int() - 127))
        out[r:r + 2048] = (value.view(part.shape[0], -1, size) * factor.unsqueeze(-1)).view(part.shape)
    return out


def _linear(x, w, bias, layout, x_scale=None):
    """The linear layer on what x (dense) and w (dense) are stored as."""
    if layout == "nvfp4":
        xs, ws = _dynamic_scale(x) if x_scale is None else x_scale, _dynamic_scale(w)
        y = _stored(x, layout, xs) @ _stored(w, layout, ws).T
    else:
        y = _stored(x, layout) @ _stored(w, layout).T
    return y if bias is None else y.add_(bias.double())


def _rounded_gelu(h, dtype):
    """GELU (tanh form) between the two layers of an MLP: from and to the layers' type."""
    out = torch.empty(h.shape, dtype=dtype, device=h.device)
    for r in range(0, h.shape[0], 2048):
        out[r:r + 2048] = torch.nn.functional.gelu(h[r:r + 2048].to(dtype).double(), approximate="tanh").to(dtype)
    return out


def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind, layout, dtype = case["kind"], case["layout"], DTYPE[case["dtype"]]
    m, n, k, with_bias = case["m"], case["n"], case["k"], case["bias"]
    with torch.inference_mode():
        if kind in ("quantize", "dequantize"):
            x = _weight(gen, m, k, dtype)
            if kind == "dequantize":
                return _stored(x, layout, _dynamic_scale(x) if layout == "nvfp4" else None)
            if layout == "nvfp4":
                scale = _scale(x) if case["static"] else _dynamic_scale(x)
                parts = [_nvfp4(x[r:r + 2048], scale) for r in range(0, m, 2048)]
                codes = torch.cat([(c[:, 0::2] << 4) | c[:, 1::2] for c, _ in parts])
                codes = torch.nn.functional.pad(codes, (0, 0, 0, -m % 16))
                return codes, _tiled(torch.cat([b.view(torch.uint8) for _, b in parts])), scale.double()
            parts = [_mxfp8(x[r:r + 2048]) for r in range(0, m, 2048)]
            data = torch.cat([d.view(torch.uint8) for d, _ in parts])
            return torch.nn.functional.pad(data, (0, 0, 0, -m % 32)), _tiled(torch.cat([e for _, e in parts]))
        x = _activation(gen, m, k, dtype)
        x_scale = _scale(x) if case["static"] and kind != "gemm" else None
        if kind == "mlp":
            fc1, fc2 = _dense_linear(gen, n, k, dtype, with_bias), _dense_linear(gen, k, n, dtype, with_bias)
            # the calibration's hidden scale and the pass's own hidden tensor, each rounded where the layers round
            sample = _rounded_gelu(_linear(x[:1024], fc1.weight, fc1.bias, layout, x_scale), dtype)
            hidden = _rounded_gelu(_linear(x, fc1.weight, fc1.bias, layout, x_scale), dtype)
            return _linear(hidden, fc2.weight, fc2.bias, layout, _dynamic_scale(sample))
        lin = _dense_linear(gen, n, k, dtype, with_bias)
        return _linear(x, lin.weight, lin.bias, layout, x_scale)
