"""What a program built on this package spends its time on, as cases that can be timed one by one.

Five kinds of work, each through the calls that a user's program makes:

* `roundtrip`: MinMaxUInt8 compression of a gradient buffer and its decompression
  (`BaguaTensorPy.compress` / `decompress_from`), what a program with a transport of its own calls;
* `bucket`: tensors marked ready, scheduled, communicated and waited for through the engine
  (`BaguaCommBackendPy`, `BaguaBucketPy`), on a communicator of one rank: the engine's own share of
  a step, without a wire.  `full` moves scattered gradients into the bucket's staging buffer and
  back, `bytegrad` also quantises and reduces them;
* `update`: what is done to weights after the exchange: the optimizer step on flat buckets, and the
  averaging steps of the decentralized algorithms;
* `block`: forward and backward of a fused convolution block on bf16 channels-last activations;
* `train`: one whole training step through `with_bagua` (zero the gradients, forward, backward with
  the bucket hooks, optimizer step).

A case is a dict of plain values.  `listed()` names the fixed ones, `draw()` gives others of the same
ranges.  One process drives one GPU.
"""
from __future__ import annotations

import dataclasses
import os

import torch
import torch.nn.functional as F

os.environ.setdefault("LOG_LEVEL", "ERROR")
os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
os.environ.setdefault("MASTER_PORT", "29517")

import bagua_core as bc  # noqa: E402
import bagua_core_b200.ops as ops  # noqa: E402
import bagua_core_b200.parallel as P  # noqa: E402
from bagua_core_b200 import models  # noqa: E402
from bagua_core_b200.ops import fused_conv, shadow, wgrad  # noqa: E402

DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
ESIZE = {"float32": 4, "float16": 2, "bfloat16": 2}
MIB = 1 << 20

# As bench.py runs: linear layers add their weight gradients in place.  (The convolution library chooses
# its kernels by rule, not by timing them as there: a choice that differs between two runs changes the
# gradients more than anything in this package may.)
torch.backends.cuda.matmul.allow_tf32 = True
torch.backends.cudnn.allow_tf32 = True
wgrad.enabled = True

# The convolution blocks of the VGG-16 in models/vision.py: (input channels, output channels, height
# and width of the input, whether a 2x2 pooling follows).
VGG_BLOCKS = [(3, 64, 224, False), (64, 64, 224, True), (64, 128, 112, False), (128, 128, 112, True),
              (128, 256, 56, False), (256, 256, 56, True), (256, 512, 28, False), (512, 512, 28, True),
              (512, 512, 14, True)]


def listed():
    return [
        # one small layer's gradient: launches and host calls
        {"name": "roundtrip_small", "kind": "roundtrip", "dtype": "float32", "chunk": 4096, "chunks": 1},
        # the default 10 MB bucket, one chunk per rank of an 8-GPU node
        {"name": "roundtrip_bucket", "kind": "roundtrip", "dtype": "float32", "chunk": 10 * MIB // 4 // 8, "chunks": 8},
        # a half-precision buffer that nothing was padded for: odd chunks, unaligned payloads
        {"name": "roundtrip_ragged", "kind": "roundtrip", "dtype": "float16", "chunk": 349527, "chunks": 3},
        # the gradient of VGG-16's first classifier layer (4096 x 25088), the largest tensor in a bucket
        {"name": "roundtrip_large", "kind": "roundtrip", "dtype": "float32", "chunk": 4096 * 25088 // 8, "chunks": 8},
        # ResNet-50's gradients in half precision left where the framework allocated them: every bucket is staged
        {"name": "bucket_staged", "kind": "bucket", "op": "full", "dtype": "float16", "tensors": "resnet50",
         "scale": 1, "bucket_mb": 10, "flat": False},
        # the same buckets' low-precision op on flat fp32 storage, as `with_bagua` lays them out
        {"name": "bucket_bytegrad", "kind": "bucket", "op": "bytegrad", "dtype": "float32", "tensors": "resnet50",
         "scale": 1, "bucket_mb": 10, "flat": True},
        # optimizer step over ResNet-50's 25.6 M parameters, with the bf16 copies a bf16 model reads
        {"name": "update_sgd", "kind": "update", "op": "sgd", "elements": 25557032, "bucket_mb": 10, "shadow": True,
         "nesterov": False, "weight_decay": 1e-4},
        # one round of asynchronous model averaging over the same weights
        {"name": "update_async", "kind": "update", "op": "async", "elements": 25557032, "dtype": "float32"},
        # the block of VGG-16 with the largest activation, at the benchmark's batch of 32
        {"name": "block_pool", "kind": "block", "c_in": 64, "c_out": 64, "size": 224, "pool": True, "batch": 32},
        # the small model of the tests and the CPU configuration: a step is all host work and launches
        {"name": "train_mlp", "kind": "train", "model": "mlp", "batch": 64, "width": 128, "depth": 3,
         "algorithm": "gradient_allreduce", "bucket_mb": 1},
        # the headline benchmark's step
        {"name": "train_vgg16", "kind": "train", "model": "vgg16", "batch": 32, "algorithm": "gradient_allreduce",
         "bucket_mb": 10},
        # BERT-large's layers, batch 8 of 384 tokens.  Two of its 24, dropout off and gradients unquantised, so
        # that a step can be compared: the library's attention backward does not repeat its bits, and depth and
        # quantisation magnify that
        {"name": "train_bert", "kind": "train", "model": "bert", "batch": 8, "seq": 384, "layers": 2,
         "algorithm": "gradient_allreduce", "bucket_mb": 64},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["roundtrip", "roundtrip", "roundtrip", "bucket", "bucket", "update", "update", "block", "train"])
    dtype = rng.choice(list(DTYPES))
    if kind == "roundtrip":
        chunks = rng.choice([1, 2, 3, 4, 8])
        total = _log(rng, 1024, 100_000_000)
        chunk = max(1, total // chunks)
        if rng.random() < 0.6:  # most buffers are padded to whole vectors per rank, as buckets are
            chunk = (chunk + 15) // 16 * 16
        return {"kind": kind, "dtype": dtype, "chunk": chunk, "chunks": chunks}
    if kind == "bucket":
        op = rng.choice(["full", "full", "bytegrad"])
        return {"kind": kind, "op": op, "dtype": dtype, "tensors": rng.choice(["resnet50", "vgg16", "mlp"]),
                "scale": rng.choice([1, 1, 2, 4]), "bucket_mb": rng.choice([1, 5, 10, 25]),
                "flat": op == "bytegrad" and rng.random() < 0.7}
    if kind == "update":
        op = rng.choice(["sgd", "sgd", "async", "average"])
        n = _log(rng, 4096, 130_000_000)
        if op == "sgd":
            return {"kind": kind, "op": op, "elements": n, "bucket_mb": rng.choice([1, 5, 10, 25]),
                    "shadow": rng.random() < 0.5, "nesterov": rng.random() < 0.3,
                    "weight_decay": rng.choice([0.0, 1e-4])}
        return {"kind": kind, "op": op, "elements": n, "dtype": "float32" if op == "async" else dtype}
    if kind == "block":
        c_in, c_out, size, pool = rng.choice(VGG_BLOCKS[1:])
        return {"kind": kind, "c_in": c_in, "c_out": c_out, "size": size, "pool": pool, "batch": _log(rng, 1, 32)}
    model = rng.choice(["mlp", "mlp", "vgg16", "bert"])
    if model == "mlp":
        return {"kind": kind, "model": model, "batch": _log(rng, 8, 512), "width": 16 * _log(rng, 4, 256),
                "depth": rng.choice([2, 3, 4, 6]), "algorithm": rng.choice(["gradient_allreduce", "bytegrad"]),
                "bucket_mb": rng.choice([1, 10])}
    if model == "vgg16":
        return {"kind": kind, "model": model, "batch": _log(rng, 2, 31), "algorithm": "gradient_allreduce",
                "bucket_mb": rng.choice([5, 10, 25])}
    return {"kind": kind, "model": model, "batch": _log(rng, 1, 8), "seq": 16 * rng.randint(2, 24),
            "layers": rng.randint(1, 2), "algorithm": "gradient_allreduce", "bucket_mb": rng.choice([25, 64])}


# ---- shapes ---------------------------------------------------------------------------------------
def _resnet50_sizes():
    sizes = [64 * 3 * 49, 64, 64]
    c = 64
    for width, blocks in ((64, 3), (128, 4), (256, 6), (512, 3)):
        for b in range(blocks):
            sizes += [width * c, width, width, width * width * 9, width, width, 4 * width * width, 4 * width, 4 * width]
            if b == 0:
                sizes += [4 * width * c, 4 * width, 4 * width]
            c = 4 * width
    return sizes + [1000 * 2048, 1000]


def _vgg16_sizes():
    sizes, c = [], 3
    for v in (64, 64, 128, 128, 256, 256, 256, 512, 512, 512, 512, 512, 512):
        sizes += [v * c * 9, v]
        c = v
    return sizes + [4096 * 25088, 4096, 4096 * 4096, 4096, 1000 * 4096, 1000]


def _tensor_sizes(case):
    """Elements of every gradient of a bucket case, in the order in which backward produces them."""
    names = {"resnet50": _resnet50_sizes, "vgg16": _vgg16_sizes,
             "mlp": lambda: [64 * 128, 128, 128 * 128, 128, 128 * 10, 10]}
    return [max(1, n // case["scale"]) for n in reversed(names[case["tensors"]]())]


def _split(sizes, esize, bucket_mb):
    """The package's greedy rule: consecutive tensors up to the bucket size."""
    groups, cur, used = [], [], 0
    for n in sizes:
        if cur and used + n * esize > bucket_mb * MIB:
            groups.append(cur)
            cur, used = [], 0
        cur.append(n)
        used += n * esize
    return groups + [cur]


def _merge(groups, most):
    """At most `most` groups: a model with many more buckets than that is given larger ones."""
    while len(groups) > most:
        groups = [sum(groups[i:i + 2], []) for i in range(0, len(groups), 2)]
    return groups


# ---- preparation ----------------------------------------------------------------------------------
_pg = None


def _process_group():
    """The process group of this process, with a scheduler of its own for every caller: one process
    holds several models here, where a user's program holds one."""
    global _pg
    if _pg is None:
        _pg = P.init_process_group(torch.device("cuda", 0))
    return dataclasses.replace(_pg, backend=bc.BaguaCommBackendPy(100, 0))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _gradient(n, dtype, gen):
    """Values like a layer's gradient: centred, small, a few far from the rest."""
    x = torch.randn(n, device="cuda", generator=gen)
    return (x * x.abs() * 1e-2).to(dtype)


def _prepare_roundtrip(case, seed):
    x = _gradient(case["chunk"] * case["chunks"], DTYPES[case["dtype"]], _gen(seed))
    out = torch.empty_like(x)
    return {"x": x, "out": out, "src": bc.BaguaTensorPy(x, "x"), "dst": bc.BaguaTensorPy(out, "out"), "chunks": case["chunks"]}


def _prepare_bucket(case, seed):
    dtype, gen = DTYPES[case["dtype"]], _gen(seed)
    groups = _merge(_split(_tensor_sizes(case), ESIZE[case["dtype"]], case["bucket_mb"]), 32)
    backend = bc.BaguaCommBackendPy(100, 0)
    stream = torch.cuda.Stream(priority=-1)
    comm = bc.BaguaSingleCommunicatorPy(0, 1, 0, stream.cuda_stream, "solo")
    values, order, buckets = [], [], []
    for i, sizes in enumerate(groups):
        # flat: back to back and padded to whole vectors; otherwise each tensor on a 512-byte boundary of its
        # own, as the framework's allocator places them.  `buffer` holds all of them either way.
        step = 1 if case["flat"] else 512 // ESIZE[case["dtype"]]
        at = [0]
        for n in sizes:
            at.append(at[-1] + (n + step) // step * step if step > 1 else at[-1] + n)
        used = at[-1]
        buffer = _gradient((used + 15) // 16 * 16, dtype, gen)
        parts = [buffer[a:a + n] for a, n in zip(at, sizes)]
        pad = buffer.numel() - used if case["flat"] else 0
        values.append(buffer)
        named = [bc.BaguaTensorPy(t, "b%d_t%d" % (i, k)) for k, t in enumerate(parts)]
        order.append(named)
        if pad:
            named = named + [bc.BaguaTensorPy(buffer[used:], "bagua_padding_tensor_bucket_%d" % i)]
        bucket = bc.BaguaBucketPy("bucket_%d" % i, named)
        bucket.append_centralized_synchronous_op(comm, None, hierarchical=False, average=True, scattergather=True,
                                                 compression="MinMaxUInt8" if case["op"] == "bytegrad" else None)
        buckets.append(bucket)
    backend.register_ordered_buckets(buckets)
    return {"backend": backend, "comm": comm, "stream": stream, "order": order, "buckets": buckets, "values": values,
            "events": [torch.cuda.Event() for _ in groups]}


def _prepare_update(case, seed):
    gen, n = _gen(seed), case["elements"]
    if case["op"] != "sgd":
        dtype = DTYPES[case["dtype"]]
        t = torch.randn(n, device="cuda", generator=gen).mul_(0.02).to(dtype)
        peer = (t.float() + 1e-3 * torch.randn(n, device="cuda", generator=gen)).to(dtype)
        return {"op": case["op"], "t": t, "peer": peer, "reduced": (4 * t.float()).to(dtype)}
    per = case["bucket_mb"] * MIB // 4
    sizes = [per] * (n // per) + ([n % per] if n % per else [])
    sizes = [sum(g) for g in _merge([[s] for s in sizes], 16)]
    module = torch.nn.Module()
    for i, s in enumerate(sizes):
        module.register_parameter("w%d" % i, torch.nn.Parameter(torch.randn(s, device="cuda", generator=gen) * 0.02))
    opt = P.FlatSGD(module.parameters(), lr=0.01, momentum=0.9, weight_decay=case["weight_decay"],
                    nesterov=case["nesterov"], bf16_shadow=case["shadow"])
    bagua = P.with_bagua(module, [opt], P.GradientAllReduceAlgorithm(), process_group=_process_group(),
                         bucket_bytes=case["bucket_mb"] * MIB)
    params = list(module.parameters())
    for p in params:
        p.grad.copy_(_gradient(p.numel(), torch.float32, gen))
    return {"op": "sgd", "opt": opt, "bagua": bagua, "params": params}


def _prepare_block(case, seed):
    gen = _gen(seed)
    torch.manual_seed(seed)
    cls = fused_conv.ConvBiasReLUPool if case["pool"] else fused_conv.ConvBiasReLU
    with torch.device("cuda"):
        m = cls(case["c_in"], case["c_out"], 3, padding=1)
    torch.nn.init.kaiming_normal_(m.weight, mode="fan_out", nonlinearity="relu", generator=gen)
    torch.nn.init.normal_(m.bias, 0, 0.05, generator=gen)
    m = m.to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    b, s = case["batch"], case["size"]
    o = s // 2 if case["pool"] else s

    def nhwc(c, hw):
        return torch.randn(b, hw, hw, c, device="cuda", generator=gen, dtype=torch.bfloat16).permute(0, 3, 1, 2)

    return {"m": m, "x": nhwc(case["c_in"], s).requires_grad_(), "dy": nhwc(case["c_out"], o) * 1e-2}


def _prepare_train(case, seed):
    gen = _gen(seed)
    torch.manual_seed(seed)
    pg = _process_group()
    b, lr = case["batch"], 0.01
    with torch.device("cuda"):
        if case["model"] == "vgg16":
            net = models.VGG16(fused_ops=True).to(memory_format=torch.channels_last)
            x = torch.randn(b, 3, 224, 224, generator=gen).contiguous(memory_format=torch.channels_last)
            y = torch.randint(0, 1000, (b,), generator=gen)
        elif case["model"] == "bert":
            net = models.BertForQuestionAnswering(models.BertConfig(layers=case["layers"], dropout=0.0))
            x = torch.randint(0, 30522, (b, case["seq"]), generator=gen)
            y = torch.randint(0, case["seq"], (b, 2), generator=gen)
            lr = 1e-4
        else:
            net = models.MLP(64, case["width"], 10, depth=case["depth"])
            x = torch.randn(b, 64, generator=gen)
            y = torch.randint(0, 10, (b,), generator=gen)
    opt = P.FlatSGD(net.parameters(), lr=lr, momentum=0.9)
    algo = P.ByteGradAlgorithm() if case["algorithm"] == "bytegrad" else P.GradientAllReduceAlgorithm()
    bagua = P.with_bagua(net, [opt], algo, process_group=pg, bucket_bytes=case["bucket_mb"] * MIB)
    grads = [bk.flattened for bk in bagua.bagua_buckets]
    # the weights lie in flat buffers of the buckets' layout: one view over each
    weights = []
    for bk in bagua.bagua_buckets:
        p = bk.tensors[0].owner.detach()
        weights.append(torch.as_strided(p, (bk.flattened.numel(),), (1,), p.storage_offset()))
    return {"net": bagua, "opt": opt, "x": x, "y": y, "grads": grads, "weights": weights, "model": case["model"]}


def prepare(case, seed):
    make = {"roundtrip": _prepare_roundtrip, "bucket": _prepare_bucket, "update": _prepare_update,
            "block": _prepare_block, "train": _prepare_train}[case["kind"]]
    state = make(case, seed)
    state["kind"] = case["kind"]
    return state


# ---- one pass -------------------------------------------------------------------------------------
def _run_roundtrip(s):
    compressed = s["src"].compress("MinMaxUInt8", s["chunks"], -1)
    s["dst"].decompress_from("MinMaxUInt8", s["chunks"], compressed)
    return s["out"]


def _run_bucket(s):
    mark = s["backend"].mark_communication_ready
    for named, event in zip(s["order"], s["events"]):
        for t in named[:-1]:
            mark(t, 0)
        event.record()  # with the bucket's last gradient
        mark(named[-1], event.cuda_event)
    s["backend"].wait_pending_comm_ops()
    torch.cuda.current_stream().wait_stream(s["stream"])
    return s["values"]


def _run_update(s):
    if s["op"] == "async":
        return ops.async_model_average(s["t"], s["reduced"], s["peer"], 4)
    if s["op"] == "average":
        return ops.average_inplace(s["t"], s["peer"])
    s["opt"].step()
    copies = [shadow.lookup(p) for p in s["params"]] if s["opt"].bf16_shadow else []
    return [p.detach() for p in s["params"]] + copies


def _run_block(s):
    x, m = s["x"], s["m"]
    x.grad = m.weight.grad = m.bias.grad = None
    y = m(x)
    y.backward(s["dy"])
    return {"y": y.detach(), "dx": x.grad, "dw": m.weight.grad, "db": m.bias.grad}


def _run_train(s):
    s["opt"].zero_grad(set_to_none=False)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        if s["model"] == "bert":
            loss = s["net"](s["x"], s["y"][:, 0], s["y"][:, 1])
        else:
            out = s["net"](s["x"])
    if s["model"] != "bert":
        loss = F.cross_entropy(out.float(), s["y"])
    loss.backward()
    s["opt"].step()
    return {"loss": loss.detach(), "grads": s["grads"], "weights": s["weights"]}


def run(state):
    return {"roundtrip": _run_roundtrip, "bucket": _run_bucket, "update": _run_update, "block": _run_block,
            "train": _run_train}[state["kind"]](state)


# ---- what a pass cannot do without ----------------------------------------------------------------
def _conv_flops(c_in, c_out, size, batch):
    return 2.0 * 9 * c_in * c_out * size * size * batch


def work(case):
    kind = case["kind"]
    if kind == "roundtrip":
        n, e = case["chunk"] * case["chunks"], ESIZE[case["dtype"]]
        return {"bytes": n * (e + 1 + 1 + e), "flops": 8 * n}
    if kind == "bucket":
        n, e = sum(_tensor_sizes(case)), ESIZE[case["dtype"]]
        # one rank: every gradient is read and written; ByteGrad quantises twice on the way
        return {"bytes": 2 * n * e, "flops": (18 if case["op"] == "bytegrad" else 0) * n}
    if kind == "update":
        n = case["elements"]
        if case["op"] == "sgd":
            return {"bytes": n * (20 + (2 if case["shadow"] else 0)), "flops": 6 * n}
        e = ESIZE[case["dtype"]]
        return {"bytes": n * e * (4 if case["op"] == "async" else 3), "flops": 3 * n}
    if kind == "block":
        c_in, c_out, s, b = case["c_in"], case["c_out"], case["size"], case["batch"]
        pixels, out = b * s * s, b * s * s // (4 if case["pool"] else 1)
        # x in, dx out; y out, dy in; weight and bias in, their gradients out
        return {"bytes": 2 * (2 * pixels * c_in + 2 * out * c_out + 2 * (9 * c_in + 1) * c_out),
                "flops": 3 * _conv_flops(c_in, c_out, s, b)}
    if case["model"] == "vgg16":
        params, b = sum(_vgg16_sizes()), case["batch"]
        c, hw, flops = 3, 224, 0.0
        for v in (64, 64, 0, 128, 128, 0, 256, 256, 256, 0, 512, 512, 512, 0, 512, 512, 512, 0):
            if v:
                flops += (2 if c == 3 else 3) * _conv_flops(c, v, hw, b)  # no gradient for the images
                c = v
            else:
                hw //= 2
        flops += 3 * 2.0 * b * (25088 * 4096 + 4096 * 4096 + 4096 * 1000)
    elif case["model"] == "bert":
        h, ffn, t = 1024, 4096, case["batch"] * case["seq"]
        layer = 4 * h * h + 2 * h * ffn
        params = case["layers"] * (layer + 9 * h + ffn) + (30522 + 512 + 2 + 2) * h + 2 * h + 2
        flops = 3 * 2.0 * t * (case["layers"] * (layer + 2 * case["seq"] * h) + 2 * h)
    else:
        dims = [64] + [case["width"]] * (case["depth"] - 1) + [10]
        params = sum(a * b + b for a, b in zip(dims, dims[1:]))
        flops = 3 * 2.0 * case["batch"] * params
    # weights and momentum read and written, the gradient written
    return {"bytes": 20.0 * params, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "roundtrip" or (kind == "bucket" and case["op"] == "full"):
        return "exact"  # quantised values are whole numbers on a grid that min and max fix; copies are copies
    if kind == "bucket":
        return {"rel": 1e-5 if case["dtype"] == "float32" else 1e-2, "max": 0.9}
    if kind == "update":
        return {"rel": 1e-5 if case.get("dtype", "float32") == "float32" else 1e-2}
    if kind == "block":
        return {"rel": 1e-2, "max": 0.5}
    # autocast: activations and their gradients are bf16 in every layer, whatever type the outputs have
    return {"rel": 2e-2, "max": 0.9}
