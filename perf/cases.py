"""Performance cases of the serving framework: models, their layers, single operators, the copy engine and an app.

A case is a dict of plain values.  ``prepare`` makes inputs, weights and the plan that a serving process keeps (buffers,
captured graphs, copy lists), ``run`` makes one pass through the package's public calls, ``exact`` is the same result in
64-bit arithmetic.  Models and layer chains run as captured CUDA graphs, as ``serving.engine`` runs them (one graph per
batch size); single operators are called directly.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from splitrpc_b200 import _C, ops
from splitrpc_b200.models import BertClassifier, ResNet50
from splitrpc_b200.models.bert import BERT_BASE

DEV = "cuda:0"
# ResNet-50 stages: width, blocks, stride of the first block, side of the incoming image
STAGES = ((64, 3, 1, 56), (128, 4, 2, 56), (256, 6, 2, 28), (512, 3, 2, 14))
HEADS = {768: 12, 1024: 16}
FRAG = 8192                                  # the wire's MTU: payload bytes of one fragment
LSTM_L, LSTM_T, LSTM_H = 8, 8, 256           # the served LSTM: layers, steps, hidden size


def listed() -> list[dict]:
    return [
        # The headline: one full dynamic batch of ResNet-50 requests behind one ingress.
        {"name": "resnet50_64", "kind": "resnet50", "batch": 64},
        # BERT-base at the served batch of 32 sequences of 128 tokens.
        {"name": "bert_base_32x128", "kind": "bert", "batch": 32, "seq": 128},
        # A residual block in the middle of the network at the full batch (the most frequent block of ResNet-50).
        {"name": "block_14px_64", "kind": "block", "stage": 2, "first": False, "batch": 64},
        # The first block of the last stage (stride 2, projection shortcut) at an odd batch that a light load forms.
        {"name": "block_7px_proj_5", "kind": "block", "stage": 3, "first": True, "batch": 5},
        # From the request's fp32 pixels to the pooled stem activations, at half the full batch.
        {"name": "stem_32", "kind": "stem", "batch": 32},
        # The classifier head of the full batch: pooling, 1000-way linear layer, softmax written as the response.
        {"name": "head_64", "kind": "head", "batch": 64},
        # One encoder layer for a single short request: the latency end, where launches count.
        {"name": "encoder_768_1x128", "kind": "encoder", "hidden": 768, "batch": 1, "seq": 128},
        # One encoder layer of BERT-large at its benchmark batch (16 sequences of 384 tokens).
        {"name": "encoder_1024_16x384", "kind": "encoder", "hidden": 1024, "batch": 16, "seq": 384},
        # The largest plain product, bound by the tensor cores.
        {"name": "gemm_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "act": "none", "residual": False, "fp32": False},
        # A ragged product with every epilogue term, as a user's own layer might have it.
        {"name": "gemm_ragged", "kind": "gemm", "m": 1003, "n": 584, "k": 1032, "act": "gelu", "residual": True, "fp32": False},
        # 64 image requests gathered from their 8 KB fragments in device memory into contiguous ring slots.
        {"name": "gather_64x602112", "kind": "gather", "requests": 64, "bytes": 602112, "shift": 0},
        # A batch of LSTM requests through the app's synchronous batch call (launch and wait, as the worker does it).
        {"name": "lstm_4", "kind": "lstm", "batch": 4},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["resnet50", "bert", "block", "block", "stem", "head", "encoder", "encoder", "gemm", "gemm", "gather", "lstm"])
    if kind == "resnet50":
        return {"kind": kind, "batch": _log_int(rng, 1, 64)}
    if kind == "bert":
        seq = rng.choice([128, 384])
        return {"kind": kind, "batch": _log_int(rng, 1, 4096 // seq), "seq": seq}
    if kind == "block":
        return {"kind": kind, "stage": rng.randrange(4), "first": rng.random() < 0.4, "batch": _log_int(rng, 1, 64)}
    if kind in ("stem", "head"):
        return {"kind": kind, "batch": _log_int(rng, 1, 64)}
    if kind == "encoder":
        seq = rng.choice([128, 384])
        return {"kind": kind, "hidden": rng.choice([768, 1024]), "batch": _log_int(rng, 1, 6144 // seq), "seq": seq}
    if kind == "gemm":
        fp32 = rng.random() < 0.25
        return {"kind": kind, "m": _log_int(rng, 1, 8192), "n": 8 * _log_int(rng, 1, 1024), "k": 8 * _log_int(rng, 4, 1024),
                "act": rng.choice(["none", "relu", "gelu"]), "residual": not fp32 and rng.random() < 0.5, "fp32": fp32}
    if kind == "gather":
        size = _log_int(rng, 64, 602112)
        return {"kind": kind, "requests": _log_int(rng, 1, 64), "bytes": size, "shift": rng.choice([0, 0, 4, 1])}
    return {"kind": kind, "batch": _log_int(rng, 1, 16)}


# ------------------------------------------------------------------ inputs and weights (from the seed alone)
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, base=0.0, dtype=torch.float32) -> torch.Tensor:
    return (torch.randn(shape, generator=g, device=DEV) * std + base).to(dtype)


def _block_shape(c: dict) -> tuple[int, int, int, int, int, int, bool]:
    """batch, incoming side, outgoing side, incoming channels, width, stride, projection shortcut"""
    width, _, stride, side = STAGES[c["stage"]]
    cin = 64 if c["stage"] == 0 else width * 2
    if c["first"]:
        return c["batch"], side, side // stride, cin, width, stride, True
    return c["batch"], side // stride, side // stride, width * 4, width, 1, False


def _block_weights(g, cin: int, width: int, proj: bool) -> dict:
    w = {}
    for name, cout, ci, k, gain in (("c1", width, cin, 1, 1.0), ("c2", width, width, 3, 1.0), ("c3", width * 4, width, 1, 0.5),
                                    ("ds", width * 4, cin, 1, 0.5)):
        if name == "ds" and not proj:
            continue
        w[name + ".w"] = _randn(g, cout, k, k, ci, std=gain * math.sqrt(2.0 / (ci * k * k)), dtype=torch.bfloat16)
        w[name + ".b"] = _randn(g, cout, std=0.05)
    return w


def _resnet_weights(g) -> dict:
    w = {"stem.w": _randn(g, 64, 3, 7, 7, std=math.sqrt(2.0 / 147), dtype=torch.bfloat16), "stem.b": _randn(g, 64, std=0.05)}
    cin = 64
    for li, (width, n, _, _) in enumerate(STAGES):
        for bi in range(n):
            for k, v in _block_weights(g, cin, width, bi == 0).items():
                w[f"l{li}.b{bi}.{k}"] = v
            cin = width * 4
    w["fc.w"], w["fc.b"] = _randn(g, 1000, 2048, std=math.sqrt(1.0 / 2048), dtype=torch.bfloat16), _randn(g, 1000, std=0.05)
    return w


def _encoder_weights(g, h: int, ffn: int) -> dict:
    bf = torch.bfloat16
    w = {}
    for name, n, k in (("qkv", 3 * h, h), ("o", h, h), ("f1", ffn, h), ("f2", h, ffn)):
        w[name + ".w"], w[name + ".b"] = _randn(g, n, k, std=0.02, dtype=bf), _randn(g, n, std=0.02)
    for name in ("ln1", "ln2"):
        w[name + ".g"], w[name + ".b"] = _randn(g, h, std=0.02, base=1.0), _randn(g, h, std=0.02)
    return w


def _bert_weights(g) -> dict:
    h, bf = BERT_BASE.hidden, torch.bfloat16
    w = {"emb.word": _randn(g, BERT_BASE.vocab, h, std=0.02, dtype=bf), "emb.pos": _randn(g, BERT_BASE.max_pos, h, std=0.02, dtype=bf),
         "emb.type": _randn(g, 2, h, std=0.02, dtype=bf), "emb.ln.g": _randn(g, h, std=0.02, base=1.0), "emb.ln.b": _randn(g, h, std=0.02)}
    for l in range(BERT_BASE.layers):
        for k, v in _encoder_weights(g, h, BERT_BASE.ffn).items():
            w[f"l{l}.{k}"] = v
    w["pool.w"], w["pool.b"] = _randn(g, h, h, std=0.02, dtype=bf), _randn(g, h, std=0.02)
    w["cls.w"], w["cls.b"] = _randn(g, 8, h, std=0.2, dtype=bf), _randn(g, 8, std=0.1)
    return w


def _lstm_weights(g) -> list:
    """Per layer: input gates [4H, H], recurrent gates [4H, H], biases [4H] (fp32, on the host)."""
    out = []
    for _ in range(LSTM_L):
        for shape in ((4 * LSTM_H, LSTM_H), (4 * LSTM_H, LSTM_H), (4 * LSTM_H,)):
            out.append(_randn(g, *shape, std=0.08).cpu().numpy().ravel())
    return out


def _inputs(c: dict, seed: int) -> dict:
    g, kind, bf = _gen(seed), c["kind"], torch.bfloat16
    if kind == "resnet50":
        return {"w": _resnet_weights(g), "x": _randn(g, c["batch"], 3, 224, 224)}
    if kind == "bert":
        return {"w": _bert_weights(g), "ids": torch.randint(0, BERT_BASE.vocab, (c["batch"], c["seq"]), generator=g, device=DEV, dtype=torch.int32)}
    if kind == "block":
        n, h, _, cin, width, _, proj = _block_shape(c)
        return {"w": _block_weights(g, cin, width, proj), "x": torch.relu(_randn(g, n, h, h, cin)).to(bf)}
    if kind == "stem":
        return {"w": _randn(g, 64, 3, 7, 7, std=math.sqrt(2.0 / 147)), "b": _randn(g, 64, std=0.05), "x": _randn(g, c["batch"], 3, 224, 224)}
    if kind == "head":
        return {"w": _randn(g, 1000, 2048, std=math.sqrt(1.0 / 2048), dtype=bf), "b": _randn(g, 1000, std=0.05),
                "x": torch.relu(_randn(g, c["batch"], 7, 7, 2048, std=2.0)).to(bf)}
    if kind == "encoder":
        return {"w": _encoder_weights(g, c["hidden"], 4 * c["hidden"]), "x": _randn(g, c["batch"] * c["seq"], c["hidden"], dtype=bf)}
    if kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"a": _randn(g, m, k, dtype=bf), "b": _randn(g, n, k, std=1.0 / math.sqrt(k), dtype=bf), "bias": _randn(g, n, std=0.1),
                "residual": _randn(g, m, n, dtype=bf) if c["residual"] else None}
    if kind == "gather":
        # every fragment in a slot of its own, as a receive ring holds them; `shift` moves the payloads off their alignment
        n_frag = c["requests"] * math.ceil(c["bytes"] / FRAG)
        arena = torch.randint(0, 256, (n_frag, FRAG + 64), generator=g, device=DEV, dtype=torch.uint8)
        return {"arena": arena, "order": torch.randperm(n_frag, generator=g, device=DEV).cpu().tolist()}
    if kind == "lstm":
        return {"w": _lstm_weights(g), "x": _randn(g, c["batch"], LSTM_T, LSTM_H)}
    raise ValueError(kind)


# ------------------------------------------------------------------ prepare / run
class _CopyList:
    def __init__(self, items):
        self.handle = _C.sg_list_create(items)

    def __del__(self):
        _C.sg_list_destroy(self.handle)


def _captured(launch) -> torch.cuda.CUDAGraph:
    """Warm-up on a side stream, then the launches as one graph, as a serving process captures each batch size."""
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        launch()
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        launch()
    return graph


def _block_launch(c: dict, w: dict, x: torch.Tensor, bufs: tuple):
    n, h, ho, cin, width, stride, proj = _block_shape(c)
    t1, t2, out = bufs
    if proj:
        wd = torch.cat([w["c3.w"].view(width * 4, width), w["ds.w"].view(width * 4, cin)], dim=1).contiguous()
        bd = w["c3.b"] + w["ds.b"]

    def launch():
        ops.gemm(x.view(-1, cin), w["c1.w"].view(width, cin), bias=w["c1.b"], act="relu", out=t1.view(-1, width))
        ops.conv2d_nhwc(t1, w["c2.w"], bias=w["c2.b"], stride=stride, pad=1, act="relu", out=t2)
        if proj:
            ops.conv1x1_dual(t2, x, wd, bias=bd, stride2=stride, act="relu", out=out)
        else:
            ops.gemm(t2.view(-1, width), w["c3.w"].view(width * 4, width), bias=w["c3.b"], residual=x.view(-1, cin), act="relu",
                     out=out.view(-1, width * 4))

    return launch


def _encoder_launch(c: dict, w: dict, x: torch.Tensor, bufs: dict):
    batch, seq, heads = c["batch"], c["seq"], HEADS[c["hidden"]]

    def launch():
        ops.gemm(x, w["qkv.w"], bias=w["qkv.b"], out=bufs["qkv"])
        ops.attention_tc_qkv(bufs["qkv"], batch, seq, heads, out=bufs["ctx"])
        ops.gemm(bufs["ctx"], w["o.w"], bias=w["o.b"], residual=x, out=bufs["attn"])
        ops.layernorm(bufs["attn"], w["ln1.g"], w["ln1.b"], out=bufs["x1"])
        ops.gemm(bufs["x1"], w["f1.w"], bias=w["f1.b"], act="gelu", out=bufs["ffn"])
        ops.gemm(bufs["ffn"], w["f2.w"], bias=w["f2.b"], residual=bufs["x1"], out=bufs["y"])
        ops.layernorm(bufs["y"], w["ln2.g"], w["ln2.b"], out=bufs["out"])

    return launch


def _load_resnet(model: ResNet50, w: dict) -> None:
    p = model.params
    for k, v in w.items():
        if k != "stem.w":
            p[k].copy_(v)
    p["stem.w_s2d"].copy_(ops.stem_weight_s2d(w["stem.w"]))
    for name, cin, width, _, ds in model.blocks:
        if ds:
            p[name + ".c3ds.w"].copy_(torch.cat([w[name + ".c3.w"].view(width * 4, width), w[name + ".ds.w"].view(width * 4, cin)], dim=1))
            p[name + ".c3ds.b"].copy_(w[name + ".c3.b"] + w[name + ".ds.b"])


def prepare(case: dict, seed: int) -> dict:
    torch.cuda.set_device(0)
    c, kind, bf = case, case["kind"], torch.bfloat16
    d = _inputs(c, seed)
    st: dict = {"kind": kind, "case": c, "in": d}
    if kind == "resnet50":
        model = ResNet50(device=0, max_batch=c["batch"])
        _load_resnet(model, d["w"])
        d["w"] = None
        probs = torch.zeros((c["batch"], 1000), device=DEV)
        st["keep"] = model
        st["graph"] = _captured(lambda: model.forward(c["batch"], x=d["x"], out=probs))
        st["out"] = {"features": model.buf["l3.b2.out"], "logits": model.buf["logits"][: c["batch"]], "probs": probs}
    elif kind == "bert":
        model = BertClassifier(BERT_BASE, seq=c["seq"], device=0, max_batch=c["batch"])
        for k, v in d["w"].items():
            model.params[k].copy_(v)
        d["w"] = None
        probs = torch.zeros((c["batch"], BERT_BASE.num_labels), device=DEV)
        st["keep"] = model
        st["graph"] = _captured(lambda: model.forward(c["batch"], ids=d["ids"], out=probs))
        st["out"] = {"hidden": model.buf["x"], "logits": model.buf["logits"][: c["batch"], : BERT_BASE.num_labels], "probs": probs}
    elif kind == "block":
        n, h, ho, _, width, _, _ = _block_shape(c)
        bufs = tuple(torch.zeros((n, s, s, ch), dtype=bf, device=DEV) for s, ch in ((h, width), (ho, width), (ho, width * 4)))
        st["graph"] = _captured(_block_launch(c, d["w"], d["x"], bufs))
        st["out"] = {"t1": bufs[0], "t2": bufs[1], "out": bufs[2]}
    elif kind == "stem":
        n = c["batch"]
        w2 = ops.stem_weight_s2d(d["w"])
        s2d = torch.zeros((n, 115, 115, 16), dtype=bf, device=DEV)
        conv = torch.zeros((n, 112, 112, 64), dtype=bf, device=DEV)
        pool = torch.zeros((n, 56, 56, 64), dtype=bf, device=DEV)

        def launch():
            ops.stem_s2d(s2d, n, x=d["x"], mean=ops.IMAGENET_MEAN, inv_std=ops.IMAGENET_INV_STD)
            ops.stem_conv(s2d, w2, n, bias=d["b"], act="relu", out=conv)
            ops.maxpool3x3s2(conv, out=pool)

        st["keep"] = (w2, s2d, conv)
        st["graph"] = _captured(launch)
        st["out"] = {"pool": pool}
    elif kind == "head":
        n = c["batch"]
        avg = torch.zeros((n, 2048), dtype=bf, device=DEV)
        logits, probs = torch.zeros((n, 1000), device=DEV), torch.zeros((n, 1000), device=DEV)

        def launch():
            ops.global_avgpool(d["x"], out=avg)
            ops.fc_skinny(avg, d["w"], bias=d["b"], out=logits)
            ops.softmax_response(logits, n, out=probs, resp_stride=4000)

        st["graph"] = _captured(launch)
        st["out"] = {"avg": avg, "logits": logits, "probs": probs}
    elif kind == "encoder":
        t, h = d["x"].shape
        bufs = {k: torch.zeros((t, n), dtype=bf, device=DEV)
                for k, n in (("qkv", 3 * h), ("ctx", h), ("attn", h), ("x1", h), ("ffn", 4 * h), ("y", h), ("out", h))}
        st["graph"] = _captured(_encoder_launch(c, d["w"], d["x"], bufs))
        st["out"] = {"ctx": bufs["ctx"], "x1": bufs["x1"], "out": bufs["out"]}
    elif kind == "gemm":
        st["out"] = torch.zeros((c["m"], c["n"]), dtype=torch.float32 if c["fp32"] else bf, device=DEV)
    elif kind == "gather":
        ring = torch.zeros((c["requests"], c["bytes"]), dtype=torch.uint8, device=DEV)
        st["list"] = _CopyList(_gather_items(c, d, ring.data_ptr()))
        st["out"] = ring
    elif kind == "lstm":
        n, req, resp = c["batch"], LSTM_T * LSTM_H * 4, LSTM_H * 4
        _C.set_rpc_mtu(FRAG)
        app = _C.make_app("lstm", 0, req, resp, d["w"], 64, 1, n)
        base = app.req_ring[0]
        _C.memcpy_async(base, d["x"].data_ptr(), n * req, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        st["app"] = app
        st["out"] = torch.zeros((n, LSTM_H), device=DEV)
    return st


def _gather_items(c: dict, d: dict, dst: int) -> list:
    """One item per fragment: fragment f of request r lies in the arena slot that the shuffled order names."""
    per, stride, src = math.ceil(c["bytes"] / FRAG), FRAG + 64, d["arena"].data_ptr()
    items = []
    for r in range(c["requests"]):
        for f in range(per):
            n = min(FRAG, c["bytes"] - f * FRAG)
            items.append((src + d["order"][r * per + f] * stride + c["shift"], dst + r * c["bytes"] + f * FRAG, n))
    return items


def run(st: dict):
    kind = st["kind"]
    if "graph" in st:
        st["graph"].replay()
    elif kind == "gemm":
        d, act = st["in"], st["case"]["act"]
        ops.gemm(d["a"], d["b"], bias=d["bias"], residual=d["residual"], act=None if act == "none" else act, out=st["out"])
    elif kind == "gather":
        _C.sg_list_launch(st["list"].handle, 0, 0, torch.cuda.current_stream().cuda_stream)
    elif kind == "lstm":
        n, out = st["case"]["batch"], st["out"]
        _, resp = _C.local_bench(st["app"], 1, n)
        _C.memcpy_async(out.data_ptr(), resp[0], n * LSTM_H * 4, torch.cuda.current_stream().cuda_stream)
    return st["out"]


# ------------------------------------------------------------------ what a pass cannot do without
def _block_work(c: dict) -> tuple[float, float]:
    n, h, ho, cin, width, _, proj = _block_shape(c)
    wts = cin * width + 9 * width * width + 4 * width * width + (4 * width * cin if proj else 0)
    macs = n * (h * h * cin * width + ho * ho * (9 * width * width + 4 * width * width + (4 * width * cin if proj else 0)))
    acts = n * (h * h * (cin + width) + ho * ho * (width + 4 * width))
    return 2.0 * (acts + wts), 2.0 * macs


def work(case: dict) -> dict:
    c, kind = case, case["kind"]
    if kind == "resnet50":
        n = c["batch"]
        flops = 2.0 * n * (112 * 112 * 64 * 147 + 2048 * 1000)
        wbytes = 2.0 * (64 * 147 + 2048 * 1000)
        for s, (width, blocks, _, _) in enumerate(STAGES):
            for b in range(blocks):
                bc = {"stage": s, "first": b == 0, "batch": n}
                _, h, ho, cin, _, _, proj = _block_shape(bc)
                flops += _block_work(bc)[1]
                wbytes += 2.0 * (cin * width + 13 * width * width + (4 * width * cin if proj else 0))
        return {"bytes": n * (602112.0 + 2 * 49 * 2048 + 8000) + wbytes, "flops": flops}
    if kind in ("encoder", "bert"):
        h = c.get("hidden", BERT_BASE.hidden)
        t = c["batch"] * c["seq"]
        layer = 2.0 * t * 12 * h * h + 4.0 * t * c["seq"] * h
        if kind == "encoder":
            return {"bytes": 2.0 * (4 * t * h + 12 * h * h), "flops": layer}
        layers = BERT_BASE.layers
        return {"bytes": 4.0 * t + 16.0 * c["batch"] + 2.0 * (t * h + 12 * h * h * layers + min(t, BERT_BASE.vocab) * h + c["seq"] * h), "flops": layer * layers}
    if kind == "block":
        b, f = _block_work(c)
        return {"bytes": b, "flops": f}
    if kind == "stem":
        n = c["batch"]
        return {"bytes": n * (602112.0 + 2 * 56 * 56 * 64) + 2 * 64 * 147, "flops": 2.0 * n * 112 * 112 * 64 * 147}
    if kind == "head":
        n = c["batch"]
        return {"bytes": n * (2 * 49 * 2048 + 2 * 2048 + 8000.0) + 2 * 2048 * 1000, "flops": 2.0 * n * 2048 * 1000}
    if kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2.0 * (m * k + n * k + (m * n if c["residual"] else 0)) + m * n * (4.0 if c["fp32"] else 2.0) + 4.0 * n,
                "flops": 2.0 * m * n * k}
    if kind == "gather":
        return {"bytes": 2.0 * c["requests"] * c["bytes"], "flops": 0.0}
    n = c["batch"]
    return {"bytes": 4.0 * (LSTM_L * (8 * LSTM_H * LSTM_H + 4 * LSTM_H) + n * (LSTM_T + 1) * LSTM_H),
            "flops": 2.0 * n * LSTM_L * LSTM_T * 8 * LSTM_H * LSTM_H}


def tolerance(case: dict):
    """About four times the distance to the 64-bit result that was measured for these layers and data types."""
    kind = case["kind"]
    if kind == "gather":
        return "exact"
    if kind == "lstm":
        return {"rel": 2e-6}            # fp32 throughout
    if kind == "gemm":
        return {"rel": 4e-5 if case["fp32"] else 8e-3}  # fp32: the accumulator's own rounding over up to 8192 terms
    if kind == "resnet50":
        return {"rel": 3e-2}            # 53 layers of bf16 activations
    if kind == "bert":
        return {"rel": 8e-2}            # 12 layers of bf16 activations
    return {"rel": 1.2e-2}              # a few bf16 roundings one after the other


# ------------------------------------------------------------------ the same results in 64 bits
def _conv64(x, w, b, stride, pad):
    """NHWC convolution in fp64, image by image group (bounded workspace)."""
    xs, wt = x.permute(0, 3, 1, 2), w.double().permute(0, 3, 1, 2).contiguous()
    return torch.cat([F.conv2d(p.contiguous(), wt, b.double(), stride, pad) for p in xs.split(16)]).permute(0, 2, 3, 1)


def _linear64(x, w, b):
    return x @ w.double().t() + b.double()


def _block64(x, w, stride, proj):
    t1 = torch.relu(_linear64(x, w["c1.w"][:, 0, 0], w["c1.b"]))
    t2 = torch.relu(_conv64(t1, w["c2.w"], w["c2.b"], stride, 1))
    idn = _linear64(x[:, ::stride, ::stride], w["ds.w"][:, 0, 0], w["ds.b"]) if proj else x
    return t1, t2, torch.relu(_linear64(t2, w["c3.w"][:, 0, 0], w["c3.b"]) + idn)


def _stem64(x, w, b):
    y = torch.relu(torch.cat([F.conv2d(p, w.to(torch.bfloat16).double(), b.double(), 2, 3) for p in x.split(16)]))
    return F.max_pool2d(y, 3, 2, 1).permute(0, 2, 3, 1)


def _encoder64(x, w, batch, seq, heads):
    h = heads * 64
    q, k, v = (t.reshape(batch, seq, heads, 64).transpose(1, 2) for t in _linear64(x, w["qkv.w"], w["qkv.b"]).split(h, dim=1))
    ctx = (torch.softmax(q @ k.transpose(-1, -2) / 8.0, -1) @ v).transpose(1, 2).reshape(batch * seq, h)
    x1 = F.layer_norm(_linear64(ctx, w["o.w"], w["o.b"]) + x, (h,), w["ln1.g"].double(), w["ln1.b"].double(), 1e-12)
    f = F.gelu(_linear64(x1, w["f1.w"], w["f1.b"]))
    out = F.layer_norm(_linear64(f, w["f2.w"], w["f2.b"]) + x1, (h,), w["ln2.g"].double(), w["ln2.b"].double(), 1e-12)
    return ctx, x1, out


def exact(case: dict, seed: int):
    torch.cuda.set_device(0)
    c, kind = case, case["kind"]
    d = _inputs(c, seed)
    if kind == "resnet50":
        w = d["w"]
        y = _stem64(d["x"].to(torch.bfloat16).double(), w["stem.w"], w["stem.b"])
        for s, (_, blocks, stride, _) in enumerate(STAGES):
            for b in range(blocks):
                pre = f"l{s}.b{b}."
                y = _block64(y, {k[len(pre):]: v for k, v in w.items() if k.startswith(pre)}, stride if b == 0 else 1, b == 0)[2]
        logits = _linear64(y.mean((1, 2)), w["fc.w"], w["fc.b"])
        return {"features": y, "logits": logits, "probs": torch.softmax(logits, -1)}
    if kind == "bert":
        w, ids = d["w"], d["ids"].long()
        batch, seq, h = c["batch"], c["seq"], BERT_BASE.hidden
        x = w["emb.word"].double()[ids] + w["emb.pos"].double()[:seq] + w["emb.type"].double()[0]
        x = F.layer_norm(x, (h,), w["emb.ln.g"].double(), w["emb.ln.b"].double(), 1e-12).view(batch * seq, h)
        for l in range(BERT_BASE.layers):
            pre = f"l{l}."
            x = _encoder64(x, {k[len(pre):]: v for k, v in w.items() if k.startswith(pre)}, batch, seq, BERT_BASE.heads)[2]
        pooled = torch.tanh(_linear64(x.view(batch, seq, h)[:, 0], w["pool.w"], w["pool.b"]))
        logits = _linear64(pooled, w["cls.w"], w["cls.b"])[:, : BERT_BASE.num_labels]
        return {"hidden": x, "logits": logits, "probs": torch.softmax(logits, -1)}
    if kind == "block":
        _, _, _, _, _, stride, proj = _block_shape(c)
        t1, t2, out = _block64(d["x"].double(), d["w"], stride, proj)
        return {"t1": t1, "t2": t2, "out": out}
    if kind == "stem":
        mean = torch.tensor(ops.IMAGENET_MEAN, device=DEV, dtype=torch.float64).view(1, 3, 1, 1)
        inv = torch.tensor(ops.IMAGENET_INV_STD, device=DEV, dtype=torch.float64).view(1, 3, 1, 1)
        return {"pool": _stem64((d["x"].double() - mean) * inv, d["w"], d["b"])}
    if kind == "head":
        avg = d["x"].double().mean((1, 2))
        logits = _linear64(avg, d["w"], d["b"])
        return {"avg": avg, "logits": logits, "probs": torch.softmax(logits, -1)}
    if kind == "encoder":
        ctx, x1, out = _encoder64(d["x"].double(), d["w"], c["batch"], c["seq"], HEADS[c["hidden"]])
        return {"ctx": ctx, "x1": x1, "out": out}
    if kind == "gemm":
        y = d["a"].double() @ d["b"].double().t() + d["bias"].double()
        if d["residual"] is not None:
            y = y + d["residual"].double()
        return torch.relu(y) if c["act"] == "relu" else (F.gelu(y) if c["act"] == "gelu" else y)
    if kind == "gather":
        per = math.ceil(c["bytes"] / FRAG)
        frags = d["arena"][torch.tensor(d["order"], device=DEV)][:, c["shift"]:c["shift"] + FRAG]
        return frags.reshape(c["requests"], per * FRAG)[:, : c["bytes"]].contiguous()
    w = [torch.from_numpy(a).to(DEV).double() for a in d["w"]]
    seqs = d["x"].double().unbind(1)
    for l in range(LSTM_L):
        wi, wh, b = w[3 * l].view(4 * LSTM_H, LSTM_H), w[3 * l + 1].view(4 * LSTM_H, LSTM_H), w[3 * l + 2]
        h = cell = torch.zeros((c["batch"], LSTM_H), device=DEV, dtype=torch.float64)
        outs = []
        for x in seqs:
            i, gg, f, o = (x @ wi.t() + h @ wh.t() + b).split(LSTM_H, dim=1)
            cell = torch.sigmoid(f) * cell + torch.sigmoid(i) * torch.tanh(gg)
            h = torch.tanh(cell) * torch.sigmoid(o)
            outs.append(h)
        seqs = outs
    return outs[-1]
