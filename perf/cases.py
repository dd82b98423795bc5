"""The work a user of this library has it do, as cases that can be timed and compared.

A case is a dict of plain values with a `kind`:
  resnet50    the network of resnet50.forward() on the engine backend, from the images to probabilities and classes
  conv        one BlobConvolution with bias and activation
  mbv2        one MobileNetV2Block
  encoder     one transformer encoder layer (post-norm), the calls a host issues for it
  product     a matrix product in one of its three forms (plain, by the transposed second matrix, batched)
Everything runs through neoml_b200.ops / neoml_b200.resnet50 and, for the two one-pass normalisation calls that ops
does not mirror, the C ABI that neoml_b200._capi declares.
"""
from __future__ import annotations

import math

import torch

from neoml_b200 import _capi as capi
from neoml_b200 import ops, resnet50

ACT_SIGMOID_GATE = 3   # NB200_ACT_SIGMOID_GATE of the C ABI: GELU in its sigmoid form
GELU_PARAM = 1.702


def listed() -> list[dict]:
    return [
        # one photo through the classification network: an interactive request, bound by latency
        {"name": "resnet50_b1", "kind": "resnet50", "batch": 1},
        # whatever a request queue held when the GPU fell free: a batch that fills no tile evenly
        {"name": "resnet50_b21", "kind": "resnet50", "batch": 21},
        # bulk classification at the batch the benchmark uses
        {"name": "resnet50_b256", "kind": "resnet50", "batch": 256},
        # the ordinary 3x3 layer of a vision network (configuration 1)
        {"name": "conv_3x3_c64", "kind": "conv", "batch": 32, "h": 56, "w": 56, "c": 64, "k": 64, "filter": 3, "stride": 1,
         "pad": 1, "dilation": 1, "act": capi.ACT_RELU, "precision": capi.PREC_3XTF32},
        # a layer of a custom network: odd image, channel counts no vector width divides, a strided 5x5 filter
        {"name": "conv_5x5_odd", "kind": "conv", "batch": 7, "h": 93, "w": 61, "c": 30, "k": 75, "filter": 5, "stride": 2,
         "pad": 2, "dilation": 1, "act": capi.ACT_RELU, "precision": capi.PREC_3XTF32},
        # the inverted-residual block of a mobile network (configuration 2)
        {"name": "mbv2_b64_c32", "kind": "mbv2", "batch": 64, "h": 56, "w": 56, "c_in": 32, "c_exp": 192, "c_out": 32,
         "stride": 1, "act": capi.ACT_RELU},
        # a downsampling block on odd-sized images, hard-swish
        {"name": "mbv2_stride2_odd", "kind": "mbv2", "batch": 17, "h": 75, "w": 75, "c_in": 24, "c_exp": 144, "c_out": 40,
         "stride": 2, "act": capi.ACT_HSWISH},
        # a layer of a text encoder over a full batch (configuration 4), causal mask
        {"name": "encoder_b64_s512", "kind": "encoder", "batch": 64, "seq": 512, "hidden": 768, "heads": 12, "ffn": 3072},
        # the same layer for a few sequences of odd length, as a service sees them
        {"name": "encoder_b3_s197", "kind": "encoder", "batch": 3, "seq": 197, "hidden": 768, "heads": 12, "ffn": 3072},
        # a large square product (configuration 5)
        {"name": "matmul_4096", "kind": "product", "form": "plain", "batch": 1, "m": 4096, "k": 4096, "n": 4096,
         "precision": capi.PREC_3XTF32},
        # a batch of odd-sized products by a transposed second operand, with the faster arithmetic the caller may choose
        {"name": "matmul_odd_tf32", "kind": "product", "form": "transposed", "batch": 5, "m": 333, "k": 517, "n": 259,
         "precision": capi.PREC_TF32},
        # the classifier of a network for one request: the smallest call there is
        {"name": "classifier_b1", "kind": "product", "form": "linear", "batch": 1, "m": 1, "k": 2048, "n": 1000,
         "precision": capi.PREC_3XTF32},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


MAX_FLOPS = 2.0e12       # below one batch-256 pass of the network
MAX_FLOATS = 200_000_000  # of one tensor


def draw(rng) -> dict:
    while True:
        kind = rng.choice(["resnet50", "conv", "conv", "mbv2", "mbv2", "encoder", "encoder", "product", "product", "product"])
        if kind == "resnet50":
            case = {"kind": kind, "batch": _log_int(rng, 2, 240)}
        elif kind == "conv":
            c = rng.choice([3, _log_int(rng, 8, 512), 4 * _log_int(rng, 4, 128), 32 * _log_int(rng, 1, 16)])
            case = {"kind": kind, "batch": _log_int(rng, 1, 64), "h": _log_int(rng, 7, 160), "w": _log_int(rng, 7, 160), "c": c,
                    "k": rng.choice([_log_int(rng, 16, 512), 32 * _log_int(rng, 1, 16)]), "filter": rng.choice([1, 3, 3, 5, 7]),
                    "stride": rng.choice([1, 1, 2]), "dilation": 1, "act": rng.choice([capi.ACT_NONE, capi.ACT_RELU, capi.ACT_HSWISH]),
                    "precision": rng.choice([capi.PREC_3XTF32, capi.PREC_3XTF32, capi.PREC_TF32])}
            if case["filter"] == 3:
                case["dilation"] = rng.choice([1, 1, 2])
            case["pad"] = case["dilation"] * (case["filter"] // 2)
        elif kind == "mbv2":
            c_in = rng.choice([16, 24, 32, 32, 64, 96, 160])
            stride = rng.choice([1, 1, 2])
            case = {"kind": kind, "batch": _log_int(rng, 1, 64), "h": _log_int(rng, 7, 112), "c_in": c_in,
                    "c_exp": c_in * rng.choice([3, 6, 6]), "c_out": rng.choice([c_in, c_in, 16, 24, 40, 64, 96]),
                    "stride": stride, "act": rng.choice([capi.ACT_RELU, capi.ACT_RELU, capi.ACT_HSWISH])}
            case["w"] = rng.choice([case["h"], _log_int(rng, 7, 112)])
        elif kind == "encoder":
            heads = rng.choice([4, 8, 12, 16])
            case = {"kind": kind, "batch": _log_int(rng, 1, 64), "seq": _log_int(rng, 16, 512), "hidden": 64 * heads, "heads": heads,
                    "ffn": 256 * heads}
        else:
            form = rng.choice(["plain", "transposed", "linear"])
            case = {"kind": kind, "form": form, "batch": 1 if form == "linear" else rng.choice([1, _log_int(rng, 2, 96)]),
                    "m": _log_int(rng, 1 if form == "linear" else 16, 4096), "k": _log_int(rng, 16, 4096),
                    "n": _log_int(rng, 16, 4096), "precision": rng.choice([capi.PREC_3XTF32, capi.PREC_3XTF32, capi.PREC_TF32])}
            if rng.random() < 0.5:   # half of the products have the even sizes that layers usually have
                case["k"], case["n"] = (max(16, v // 16 * 16) for v in (case["k"], case["n"]))
        w = work(case)
        if w["flops"] <= MAX_FLOPS and max(_floats(case)) <= MAX_FLOATS:
            return case


# ---------------------------------------------------------------------------------------------- sizes
def _out(size: int, filt: int, pad: int, stride: int, dil: int = 1) -> int:
    return ops.conv_output_size(size, filt, pad, stride, dil)


def _floats(case: dict) -> list[int]:
    """Elements of the larger tensors of a case."""
    if case["kind"] == "resnet50":
        return [1]
    if case["kind"] == "conv":
        ho, wo = (_out(case[s], case["filter"], case["pad"], case["stride"], case["dilation"]) for s in ("h", "w"))
        return [case["batch"] * case["h"] * case["w"] * case["c"], case["batch"] * ho * wo * case["k"]]
    if case["kind"] == "mbv2":
        return [case["batch"] * case["h"] * case["w"] * case["c_exp"]]
    if case["kind"] == "encoder":
        return [case["batch"] * case["seq"] * case["ffn"], case["batch"] * case["heads"] * case["seq"] ** 2]
    return [case["batch"] * case["m"] * case["k"], case["batch"] * case["k"] * case["n"], case["batch"] * case["m"] * case["n"]]


def work(case: dict) -> dict:
    """Bytes: every input, weight and result of the pass once, fp32 (the network: each layer's too, as its layers are
    separate calls).  Flops: two per multiply-accumulate, counted once whatever the arithmetic issues."""
    kind = case["kind"]
    if kind == "resnet50":
        n = case["batch"]
        return {"bytes": resnet50.contraction_bytes_per_image() * n + resnet50.weight_bytes(), "flops": resnet50.flops_per_image() * n}
    if kind == "conv":
        n, c, k, f = case["batch"], case["c"], case["k"], case["filter"]
        ho, wo = (_out(case[s], f, case["pad"], case["stride"], case["dilation"]) for s in ("h", "w"))
        return {"bytes": 4.0 * (n * case["h"] * case["w"] * c + k * f * f * c + k + n * ho * wo * k),
                "flops": 2.0 * n * ho * wo * k * f * f * c}
    if kind == "mbv2":
        n, h, w, ci, ce, co = (case[s] for s in ("batch", "h", "w", "c_in", "c_exp", "c_out"))
        ho, wo = _out(h, 3, 1, case["stride"]), _out(w, 3, 1, case["stride"])
        return {"bytes": 4.0 * (n * h * w * ci + n * ho * wo * co + ce * (ci + 9 + co + 2) + co),
                "flops": 2.0 * n * (h * w * ci * ce + ho * wo * ce * (9 + co))}
    if kind == "encoder":
        b, s, hid, ffn = case["batch"], case["seq"], case["hidden"], case["ffn"]
        rows = b * s
        return {"bytes": 4.0 * (2 * rows * hid + 4 * hid * (hid + 1) + 2 * hid * ffn + ffn + 5 * hid + s * s),
                "flops": 2.0 * rows * hid * (4 * hid + 2 * ffn) + 4.0 * b * s * s * hid}
    b, m, k, n = (case[s] for s in ("batch", "m", "k", "n"))
    return {"bytes": 4.0 * b * (m * k + k * n + m * n), "flops": 2.0 * b * m * k * n}


def tolerance(case: dict):
    """About four times the distance from an evaluation in double precision: plain TF32 keeps 11 significant bits of its
    operands (3e-4 whatever the size); in fp32 arithmetic the tensor core's accumulation truncates, so the distance grows
    with the length of the sum (5e-7 at 16 products, 1e-5 at 4096; 3e-6 to 5e-6 for an encoder layer, 2e-5 for the whole
    network, whose classes may differ where two probabilities tie)."""
    kind = case["kind"]
    if case.get("precision") == capi.PREC_TF32:
        return {"rel": 1.2e-3}
    if kind == "resnet50":
        return {"rel": 8e-5, "differ": 0.01}
    if kind == "encoder":
        return {"rel": 2e-5}
    length = {"conv": lambda: case["filter"] ** 2 * case["c"], "mbv2": lambda: case["c_exp"], "product": lambda: case["k"]}[kind]()
    return {"rel": 2.4e-6 + 1e-8 * length}


# ---------------------------------------------------------------------------------------------- inputs
def prepare(case: dict, seed: int) -> dict:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def normal(*shape, std=1.0):
        return torch.empty(shape, device="cuda").normal_(0.0, std, generator=g)

    def uniform(*shape, low=0.0, high=1.0):
        return torch.empty(shape, device="cuda").uniform_(low, high, generator=g)

    kind = case["kind"]
    st = {"case": case}
    if kind == "resnet50":
        # He-normal filters, the folded scale of each block's last convolution, small free terms; pixels in [0, 1]
        w = {}
        for sp in resnet50.conv_specs():
            std = math.sqrt(2.0 / (sp.k * sp.k * sp.c_in)) * (resnet50.RESIDUAL_BRANCH_SCALE if sp.name.endswith("_c3") else 1.0)
            w[sp.name + ".w"] = normal(sp.c_out, sp.k, sp.k, sp.c_in, std=std)
            w[sp.name + ".b"] = uniform(sp.c_out, low=-0.1, high=0.1)
        w["fc.w"] = normal(resnet50.CLASSES, 2048, std=math.sqrt(2.0 / 2048))
        w["fc.b"] = uniform(resnet50.CLASSES, low=-0.1, high=0.1)
        st.update(backend=resnet50.EngineBackend(), weights=w, x=uniform(case["batch"], 224, 224, 3))
    elif kind == "conv":
        f, c = case["filter"], case["c"]
        st.update(x=normal(case["batch"], case["h"], case["w"], c).clamp_(min=0.0),
                  filter=normal(case["k"], f, f, c, std=math.sqrt(2.0 / (f * f * c))), bias=uniform(case["k"], low=-0.1, high=0.1))
    elif kind == "mbv2":
        ci, ce, co = case["c_in"], case["c_exp"], case["c_out"]
        st.update(x=normal(case["batch"], case["h"], case["w"], ci), expand=normal(ce, ci, std=math.sqrt(2.0 / ci)),
                  expand_bias=uniform(ce, low=-0.2, high=0.2), channelwise=normal(3, 3, ce, std=math.sqrt(2.0 / 9)),
                  channelwise_bias=uniform(ce, low=-0.2, high=0.2), down=normal(co, ce, std=math.sqrt(1.0 / ce)),
                  down_bias=uniform(co, low=-0.2, high=0.2))
    elif kind == "encoder":
        hid, ffn, seq = case["hidden"], case["ffn"], case["seq"]
        w = {}
        for name in ("q", "k", "v", "o"):
            w[name + ".w"], w[name + ".b"] = normal(hid, hid, std=0.02), uniform(hid, low=-0.1, high=0.1)
        w["ffn1.w"], w["ffn1.b"] = normal(ffn, hid, std=0.02), uniform(ffn, low=-0.1, high=0.1)
        w["ffn2.w"], w["ffn2.b"] = normal(hid, ffn, std=0.02), uniform(hid, low=-0.1, high=0.1)
        for name in ("norm1", "norm2"):
            w[name + ".scale"], w[name + ".bias"] = uniform(hid, low=0.5, high=1.5), uniform(hid, low=-0.2, high=0.2)
        st.update(x=normal(case["batch"] * seq, hid), weights=w,
                  scale=torch.full((1,), 1.0 / math.sqrt(hid // case["heads"]), device="cuda"),
                  mask=torch.triu(torch.full((seq, seq), -1e9, device="cuda"), diagonal=1))
    else:
        b, m, k, n = (case[s] for s in ("batch", "m", "k", "n"))
        if case["form"] == "linear":
            st.update(a=normal(m, k), b=normal(n, k, std=math.sqrt(1.0 / k)), bias=uniform(n, low=-0.1, high=0.1))
        else:
            st.update(a=normal(b, m, k), b=normal(*((b, n, k) if case["form"] == "transposed" else (b, k, n))))
    return st


# ---------------------------------------------------------------------------------------------- the passes
def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "resnet50":
        return resnet50.forward(state["backend"], state["weights"], state["x"])
    if kind == "conv":
        return ops.BlobConvolution(state["x"], state["filter"], state["bias"], padding=(case["pad"],) * 2,
                                   stride=(case["stride"],) * 2, dilation=(case["dilation"],) * 2, act=case["act"],
                                   precision=case["precision"])
    if kind == "mbv2":
        return ops.MobileNetV2Block(state["x"], state["expand"], state["expand_bias"], state["channelwise"],
                                    state["channelwise_bias"], state["down"], state["down_bias"], stride=case["stride"],
                                    residual=case["stride"] == 1 and case["c_in"] == case["c_out"], expand_act=case["act"],
                                    channelwise_act=case["act"])
    if kind == "encoder":
        return _encoder(case, state["x"], state["weights"], state["scale"], state["mask"])
    if case["form"] == "linear":
        return ops.MultiplyMatrixByTransposedMatrix(state["a"], state["b"], free_term=state["bias"], precision=case["precision"])
    if case["form"] == "transposed":
        return ops.BatchMultiplyMatrixByTransposedMatrix(state["a"], state["b"], precision=case["precision"])
    return ops.MultiplyMatrixByMatrix(state["a"], state["b"], precision=case["precision"])


def _normalize(x: torch.Tensor, scale: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """Object normalisation over the rows of x, eps 1e-5: the calls the normalisation layer makes, its matrix passes in
    their one-pass forms."""
    rows, width = x.shape
    lib, stream = capi.load(), torch.cuda.current_stream().cuda_stream
    neg_mean = ops.SumMatrixColumns(x, rows, width)
    ops.vector_op("NEG_MULTIPLY", neg_mean, value=1.0 / width, result=neg_mean)
    inv = torch.empty(rows, device=x.device)
    capi.check("SumMatrixColumns (shifted)", lib.nb200_sum_matrix_columns_shifted(
        stream, inv.data_ptr(), x.data_ptr(), rows, width, neg_mean.data_ptr(), 1))
    ops.vector_op("MULTIPLY", inv, value=1.0 / width, result=inv)
    ops.vector_op("ADD_VALUE", inv, value=1e-5, result=inv)
    ops.vector_op("SQRT", inv, result=inv)
    ops.vector_op("INV", inv, result=inv)
    y = torch.empty_like(x)
    capi.check("rows and columns affine", lib.nb200_matrix_rows_cols_affine(
        stream, x.data_ptr(), rows, width, neg_mean.data_ptr(), 0, inv.data_ptr(), scale.data_ptr(), bias.data_ptr(), y.data_ptr()))
    return y


def _encoder(case: dict, x: torch.Tensor, w: dict, scale: torch.Tensor, mask: torch.Tensor) -> torch.Tensor:
    b, s, hid, heads = case["batch"], case["seq"], case["hidden"], case["heads"]
    d = hid // heads
    linear = ops.MultiplyMatrixByTransposedMatrix
    q = linear(x, w["q.w"], free_term=w["q.b"])
    k = linear(x, w["k.w"], free_term=w["k.b"])
    v = linear(x, w["v.w"], free_term=w["v.b"])
    q = ops.TransposeMatrix(b, q, s, 1, heads, d).view(b * heads, s, d)
    v = ops.TransposeMatrix(b, v, s, 1, heads, d).view(b * heads, s, d)
    kt = ops.TransposeMatrix(b, k, s, 1, hid, 1).view(b * heads, d, s)
    if d == 64 and s >= 128 and s % 4 == 0:   # what the one-kernel chain covers
        ctx = ops.AttentionScoresValues(q, kt, v, scale=scale, mask=mask)
    else:
        scores = ops.MultiplyMatrixByMatrix(q, kt)
        ops.MatrixSoftmaxByRowsFused(scores, b * heads * s, s, scale=scale, row_bias=mask, bias_rows=s, result=scores)
        ctx = ops.MultiplyMatrixByMatrix(scores, v)
    ctx = ops.TransposeMatrix(b, ctx, heads, 1, s, d).view(b * s, hid)
    y = linear(ctx, w["o.w"], free_term=w["o.b"], residual=x)
    y = _normalize(y, w["norm1.scale"], w["norm1.bias"])
    h = linear(y, w["ffn1.w"], free_term=w["ffn1.b"], act=ACT_SIGMOID_GATE, act_param=GELU_PARAM)
    o = linear(h, w["ffn2.w"], free_term=w["ffn2.b"], residual=y)
    return _normalize(o, w["norm2.scale"], w["norm2.bias"])
