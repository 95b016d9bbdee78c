"""What a program that links libodla_b200 has it do, as a list of measurable cases.

A case is one HALO-style graph (the networks of ``halo_models`` and a detector's suppression step) with a storage
type, a batch and a place where the caller's buffers live.  ``prepare`` makes what such a program keeps -- the planned
computation and its own input and output buffers -- and ``run`` is one call: bind the buffers, execute.  The planned
computation is shared by the states of one case (a program compiles its model once and feeds it new inputs) and goes
away with the last of them.

    storage   f32   the library's default, no item set          f16 / bf16   ODLA_FP16_MODE / ODLA_BF16_MODE
              s8    quantise / dequantise form: ResNet-50 throughout, BERT's dense layers (the rest in f16)
    buffers   device  bound pointers are GPU memory             pinned       bound pointers are pinned host memory
              numpy   ordinary host arrays through Graph.run
"""
import ctypes
import functools
import importlib
import math
import weakref

import numpy as np
import torch

PKG = "heterogeneity-aware-lowering-and-optimization_b200"
pkg = importlib.import_module(PKG)
odla = pkg.odla
mnist = importlib.import_module(PKG + ".halo_models.mnist")
resnet50 = importlib.import_module(PKG + ".halo_models.resnet50")
yolov3 = importlib.import_module(PKG + ".halo_models.yolov3")
bert = importlib.import_module(PKG + ".halo_models.bert")

BERT_POSITIONS = 384     # rows of the position table; a graph for shorter sequences uses the first of them
F32_FLOPS = 2 * 8 * resnet50.MAC_PER_IMAGE        # the largest listed f32 case
MAX_FLOPS = 2 * 256 * resnet50.MAC_PER_IMAGE      # the largest listed case
TORCH = {odla.FLOAT32: torch.float32, odla.FLOAT16: torch.float16, odla.INT32: torch.int32, odla.INT8: torch.int8}


def listed():
    return [
        # the documentation's first example (soft-max regression, fp32, host arrays): nearly all of it is call overhead
        {"name": "classifier_b64_f32_numpy", "net": "classifier", "storage": "f32", "batch": 64, "buffers": "numpy"},
        # one image at a time, as an online service sees it
        {"name": "resnet50_b1_f16", "net": "resnet50", "storage": "f16", "batch": 1, "buffers": "device"},
        # a user who sets no item gets float storage: a small batch in full precision
        {"name": "resnet50_b8_f32", "net": "resnet50", "storage": "f32", "batch": 8, "buffers": "device"},
        # whatever a request queue had gathered: an odd batch, bf16 storage, fp32 at the boundary
        {"name": "resnet50_b45_bf16", "net": "resnet50", "storage": "bf16", "batch": 45, "buffers": "device"},
        # the benchmark's own configuration
        {"name": "resnet50_b256_f16", "net": "resnet50", "storage": "f16", "batch": 256, "buffers": "device"},
        # ... in int8 from pinned host buffers, with two sub-batches so that copies run under kernels
        {"name": "resnet50_b256_s8_pinned", "net": "resnet50", "storage": "s8", "batch": 256, "buffers": "pinned"},
        # detection: the benchmark's batch, and one large picture
        {"name": "yolov3_416_b16_f16", "net": "yolov3", "storage": "f16", "batch": 16, "size": 416, "buffers": "device"},
        {"name": "yolov3_608_b1_f16", "net": "yolov3", "storage": "f16", "batch": 1, "size": 608, "buffers": "device"},
        # suppression of a detector's candidates (three heads of a 416 x 416 picture, 80 classes)
        {"name": "nms_b1_c80_n10647", "net": "nms", "storage": "f32", "batch": 1, "classes": 80, "boxes": 10647, "buffers": "device"},
        # an encoder over full sequences, in both forms, and over a ragged few
        {"name": "bert_b64_s128_f16", "net": "bert", "storage": "f16", "batch": 64, "seq": 128, "buffers": "device"},
        {"name": "bert_b64_s128_s8", "net": "bert", "storage": "s8", "batch": 64, "seq": 128, "buffers": "device"},
        {"name": "bert_b9_s77_f16", "net": "bert", "storage": "f16", "batch": 9, "seq": 77, "buffers": "device"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    net = rng.choice(["classifier", "resnet50", "resnet50", "resnet50", "yolov3", "yolov3", "nms", "bert", "bert", "bert"])
    if net == "classifier":
        return {"net": net, "storage": rng.choice(["f32", "f16"]), "batch": _log_int(rng, 1, 4096), "buffers": "numpy"}
    if net == "nms":
        return {"net": net, "storage": "f32", "batch": rng.randint(1, 4), "classes": _log_int(rng, 1, 80), "boxes": _log_int(rng, 1000, 22743), "buffers": "device"}
    case = {"net": net, "storage": rng.choice(["f32", "f16", "f16", "bf16"] if net == "yolov3" else ["f32", "f16", "f16", "bf16", "s8", "s8"])}
    if net == "yolov3":
        case["size"] = 32 * rng.randint(10, 19)
    if net == "bert":
        case["seq"] = _log_int(rng, 16, BERT_POSITIONS)
    cap = F32_FLOPS if case["storage"] == "f32" else MAX_FLOPS
    while net == "yolov3" and _flops(dict(case, batch=1)) > cap:
        case["size"] -= 32
    most = max(1, int(cap / _flops(dict(case, batch=1))))
    case["batch"] = _log_int(rng, 1, min(most, 256))
    case["buffers"] = rng.choice(["device", "device", "device", "pinned"])
    return case


# ------------------------------------------------------------------------- work ----
def _flops(c):
    b = c["batch"]
    if c["net"] == "classifier":
        return 2 * b * mnist.MAC_PER_BATCH_ROW
    if c["net"] == "nms":
        return b * c["classes"] * c["boxes"]          # every score is looked at once
    if c["net"] == "resnet50":
        return 2 * b * resnet50.MAC_PER_IMAGE
    if c["net"] == "yolov3":
        return 2 * b * yolov3.MAC_PER_IMAGE_416 * c["size"] ** 2 // 416 ** 2
    h, f, s = bert.BASE["hidden"], bert.BASE["ffn"], c["seq"]
    return 2 * b * bert.BASE["layers"] * (s * (4 * h * h + 2 * h * f) + 2 * s * s * h)


def work(case):
    c = case
    b, e = c["batch"], {"f32": 4, "f16": 2, "bf16": 2, "s8": 1}[c["storage"]]
    io = {"f32": 4, "bf16": 4, "f16": 2, "s8": 2}[c["storage"]]      # ResNet-50's images at the boundary
    if c["net"] == "classifier":
        n = 4 * b * (784 + 10) + e * 7840
    elif c["net"] == "nms":
        n = 4 * b * c["boxes"] * (4 + c["classes"]) + 12 * _nms_rows(c)
    elif c["net"] == "resnet50":
        n = b * (224 * 224 * 3 * io + 1000 * (2 if c["storage"] == "f16" else 4)) + 25502912 * e
    elif c["net"] == "yolov3":
        weights = sum(k * k * cin * cout for _, k, cin, cout, _, _ in yolov3.conv_specs())
        cells = sum((c["size"] // s) ** 2 for s in (8, 16, 32))
        n = 4 * b * (c["size"] ** 2 * 3 + cells * 255) + weights * e
    else:
        h, f, s = bert.BASE["hidden"], bert.BASE["ffn"], c["seq"]
        table = min(b * s, bert.BASE["vocab"]) * h * (2 if c["storage"] != "f32" else 4)
        n = b * s * (4 + 4 * h) + table + bert.BASE["layers"] * (4 * h * h + 2 * h * f) * e
    return {"bytes": n, "flops": _flops(c)}


def tolerance(case):
    if case["net"] == "nms":
        return "exact"
    if case["storage"] == "f32":
        return {"rel": 2e-5}
    if case["storage"] == "s8":
        # ResNet-50's integers are exact and its soft-max is fp32; BERT quantises f16 intermediates, so that a value next
        # to a rounding boundary moves by a whole step
        return {"rel": 1e-5} if case["net"] == "resnet50" else {"rel": 0.03, "max": 0.5}
    return {"rel": 0.03 if case["storage"] == "bf16" else 0.01}


# ---------------------------------------------------------------- models and weights ----
@functools.lru_cache(maxsize=None)
def _lib():
    return pkg.load()


@functools.lru_cache(maxsize=None)
def _weights(net):
    if net == "bert":
        return bert.weights(dict(bert.BASE, seq=BERT_POSITIONS))
    return {"classifier": mnist, "resnet50": resnet50, "yolov3": yolov3}[net].weights()


@functools.lru_cache(maxsize=None)
def _int8(net):
    w = _weights(net)
    if net == "resnet50":
        return resnet50.quantize_weights(w), resnet50.calibrate(w, n_images=8)
    cfg = dict(bert.BASE, seq=128)
    return bert.quantize(cfg, dict(w, pos_emb=np.ascontiguousarray(w["pos_emb"][:, :128])), n_sequences=1)


def _nms_rows(c):
    return min(100 * c["classes"] * c["batch"], 8000)


class _Model:
    """A planned computation; closed when the last state that uses it goes."""

    def __init__(self, c):
        b, st, lib = c["batch"], c["storage"], _lib()
        half = st == "f16" or (st == "s8" and c["net"] == "bert")
        g = odla.Graph(lib, c["net"], fp16=half, bf16=st == "bf16", n_gpus=1, sub_batches=2 if c["buffers"] == "pinned" else None)
        self.graph = g
        if c["net"] == "classifier":
            mnist.build(g, b, _weights("classifier"))
        elif c["net"] == "nms":
            boxes, scores = g.Argument("boxes", (b, c["boxes"], 4)), g.Argument("scores", (b, c["classes"], c["boxes"]))
            g.Output(g.NMS(boxes, scores, 100, 0.45, 0.25, _nms_rows(c), "selected"))
        elif c["net"] == "resnet50" and st == "s8":
            wq, scales = _int8("resnet50")
            resnet50.build_int8(g, b, _weights("resnet50"), wq, scales, input_type=odla.FLOAT16)
        elif c["net"] == "resnet50":
            resnet50.build(g, b, _weights("resnet50"), input_type=odla.FLOAT16 if st == "f16" else odla.FLOAT32)
        elif c["net"] == "yolov3":
            yolov3.build(g, b, _weights("yolov3"), size=c["size"])
        else:
            w = _weights("bert")
            w = dict(w, pos_emb=np.ascontiguousarray(w["pos_emb"][:, :c["seq"]]))
            bert.build(g, b, dict(bert.BASE, seq=c["seq"]), w, quant=_int8("bert") if st == "s8" else None)
        g.context()
        exe = ctypes.c_void_p()
        if lib.CompileComputation(g.comp, None, ctypes.byref(exe)) != odla.SUCCESS:
            raise RuntimeError("odla_CompileComputation failed")

    def __del__(self):
        if hasattr(self, "graph"):
            self.graph.close()


_models = weakref.WeakValueDictionary()


def _model(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    m = _models.get(key)
    if m is None:
        m = _models[key] = _Model(case)
    return m


# ------------------------------------------------------------------------- inputs ----
def _detector_candidates(c, gen):
    """Boxes and scores as a detector leaves them: a couple of dozen objects per picture, each with a cluster of
    overlapping confident candidates, everything else background far below the threshold."""
    b, n, k = c["batch"], c["boxes"], c["classes"]
    r = functools.partial(torch.rand, generator=gen, device="cuda")
    centre, extent = r((b, n, 2)) * 416, 8 + 112 * r((b, n, 2))
    scores = 0.1 * r((b, k, n)) ** 4
    for i in range(b):
        objects, per = 24, min(40, n // 48)
        where = torch.randperm(n, generator=gen, device="cuda")[:objects * per]
        owner = torch.arange(objects, device="cuda").repeat_interleave(per)
        centre[i, where] = (r((objects, 2)) * 416)[owner] + 4 * torch.randn((objects * per, 2), generator=gen, device="cuda")
        extent[i, where] = (24 + 96 * r((objects, 2)))[owner] * (0.9 + 0.2 * r((objects * per, 2)))
        label = torch.randint(0, k, (objects,), generator=gen, device="cuda")[owner]
        scores[i, label, where] = 0.3 + 0.69 * r((objects * per,))
    return {"boxes": torch.cat([centre - extent / 2, centre + extent / 2], dim=2).contiguous(), "scores": scores}


def _inputs(c, g, seed):
    if c["net"] == "classifier":
        return mnist.inputs(c["batch"], seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if c["net"] == "nms":
        return _detector_candidates(c, gen)
    name = g.arg_names[0]
    shape, dtype = g.shapes[name], TORCH[g.dtypes[name]]
    if c["net"] == "bert":
        x = torch.randint(0, bert.BASE["vocab"], shape, generator=gen, device="cuda", dtype=dtype)
    elif c["net"] == "yolov3":
        x = torch.rand(shape, generator=gen, device="cuda", dtype=dtype)
    else:
        x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)
    return {name: x}


def prepare(case, seed):
    m = _model(case)
    g, state = m.graph, {"model": m, "buffers": case["buffers"]}
    state["in"] = _inputs(case, g, seed)
    if case["buffers"] != "numpy":
        state["out"] = {n: torch.empty(g.shapes[n], dtype=TORCH[g.dtypes[n]], device="cuda") for n in g.out_names}
    if case["buffers"] == "pinned":
        for side in ("in", "out"):
            state[side] = {n: torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for n, t in state[side].items()}
    return state


def run(state):
    g = state["model"].graph
    if state["buffers"] == "numpy":
        return g.run(state["in"])
    for n, t in state["in"].items():
        g.bind_input(n, t.data_ptr())
    for n, t in state["out"].items():
        g.bind_output(n, t.data_ptr())
    status = g.execute()
    if status != odla.SUCCESS:
        raise RuntimeError("odla_ExecuteComputation failed with odla_status %d" % status)
    return state["out"]
