"""The work this framework is used for, as cases that can be timed and compared.

Two kinds of use. A program that runs a whole graph keeps a `plan.CompiledGraph` (weights packed once, one CUDA-graph replay
per call on a stream of its own). A program that runs an execution plan node by node calls the operators of `ops`: every call
takes and returns tensors in the reference's layout (NCHW / OIHW float32, int8 for the quantized convolution) and includes
whatever conversion the operator needs. Inference is the only direction the framework has.

    family   one pass                                                            ranges
    net      CompiledGraph of ResNet-18, 3x224x224 images                        bf16 1..1024 images, tf32 1..256, tf32x3 1..64,
                                                                                 fp32 (bit-exact) 1..32
    layer    CompiledGraph of one convolution + bias + ReLU                      bf16 / tf32, 1..64 images, any channel counts
    conv     ops.nn_conv2d + bias + residual + ReLU                              tf32 / bf16 / fp32, 1..64 images, ragged sizes
    conv_s8  ops.nn_conv2d_s8, both layouts                                      1..256 images
    chain    ops.max_pool2d_add_relu                                             1..64 images, ragged planes
    head     global average pool -> flatten -> gemm -> softmax, op by op         1..1024 images

Shapes of the listed cases are those of the repository's benchmark configurations, except the ragged convolution.
"""
import math

import numpy as np
import torch

from hdkx_aicompiler_b200 import ops, plan, relay, resnet18


def listed():
    return [
        # one layer of a graph on a single small image: nothing but launches and conversions
        dict(name="layer_bf16_n1", kind="layer", precision="bf16", n=1, c=64, h=56, w=56, o=64, k=3, s=1),
        # one image as it arrives: latency of a whole network
        dict(name="resnet18_bf16_n1", kind="net", precision="bf16", n=1),
        # a server's ordinary batch, and one GPU's share of the 1024-image batch on eight GPUs
        dict(name="resnet18_bf16_n128", kind="net", precision="bf16", n=128),
        # the throughput batch
        dict(name="resnet18_bf16_n1024", kind="net", precision="bf16", n=1024),
        # batch 32 at the precisions of users who hold to the float32 reference: rounded operands, three passes, equal bits
        dict(name="resnet18_tf32_n32", kind="net", precision="tf32", n=32),
        dict(name="resnet18_tf32x3_n32", kind="net", precision="tf32x3", n=32),
        dict(name="resnet18_fp32_n32", kind="net", precision="fp32", n=32),
        # node-by-node convolution with its fused epilogue, nothing about its size convenient
        dict(name="conv_tf32_ragged", kind="conv", precision="tf32", n=9, c=72, h=45, w=51, o=120, k=3, s=1),
        # quantized layers: the reference's layout in and out, and tensors resident in the kernels' layout
        dict(name="conv_s8_nchw_n256", kind="conv_s8", nhwc=False, n=256, c=128, h=28, w=28, o=128, k=3, s=1),
        dict(name="conv_s8_nhwc_n256", kind="conv_s8", nhwc=True, n=256, c=256, h=14, w=14, o=256, k=3, s=1),
        # the memory-bound chain
        dict(name="pool_chain_n32", kind="chain", n=32, c=64, h=112, w=112),
        # a classifier's head run node by node: four small operators, host work and launches
        dict(name="head_n32", kind="head", precision="tf32", n=32, c=512, h=7, w=7, o=1000),
    ]


def _spread(rng, lo, hi):
    """A whole number of lo..hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


_NET_MOST = {"bf16": 1024, "tf32": 256, "tf32x3": 64, "fp32": 32}


def draw(rng):
    kind = rng.choice(["net", "net", "net", "layer", "conv", "conv", "conv_s8", "conv_s8", "chain", "head"])
    if kind == "net":
        precision = rng.choice(["bf16", "bf16", "tf32", "tf32x3", "fp32"])
        return dict(kind=kind, precision=precision, n=_spread(rng, 1, _NET_MOST[precision]))
    if kind == "chain":
        return dict(kind=kind, n=_spread(rng, 1, 64), c=_spread(rng, 3, 128), h=_spread(rng, 14, 112), w=_spread(rng, 14, 112))
    if kind == "head":
        h = rng.randint(4, 9)
        return dict(kind=kind, precision=rng.choice(["tf32", "bf16"]), n=_spread(rng, 1, 1024), c=_spread(rng, 64, 1024), h=h, w=h,
                    o=_spread(rng, 10, 2000))
    while True:
        k, s = rng.choice([(3, 1), (3, 1), (3, 2), (1, 1), (1, 2)])
        case = dict(kind=kind, h=_spread(rng, 7, 112), w=0, k=k, s=s)
        case["w"] = max(7, case["h"] + rng.randint(-3, 3))
        if kind == "conv_s8":
            nhwc = rng.random() < 0.5
            case.update(nhwc=nhwc, n=_spread(rng, 1, 256))
            # the resident layout holds whole channel blocks; the reference's layout takes any count
            case.update(c=rng.choice([32, 64, 128, 256, 512]) if nhwc else _spread(rng, 16, 512),
                        o=16 * rng.randint(2, 32) if nhwc else _spread(rng, 16, 512))
        else:
            case.update(precision=rng.choice(["tf32", "bf16"] + (["fp32"] if kind == "conv" else [])), n=_spread(rng, 1, 64),
                        c=_spread(rng, 16, 512), o=_spread(rng, 16, 512))
        most = 3e10 if case.get("precision") == "fp32" else 1e11
        if _conv_flops(case) <= most:
            return case


def _out_hw(case):
    """Same-style padding k // 2."""
    return tuple((case[d] + 2 * (case["k"] // 2) - case["k"]) // case["s"] + 1 for d in ("h", "w"))


def _conv_flops(case):
    oh, ow = _out_hw(case)
    return 2.0 * case["n"] * oh * ow * case["o"] * case["c"] * case["k"] ** 2


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _conv_tensors(case, seed):
    """The distributions of the benchmark's single convolution: images U(-1,1), Kaiming-scaled filters, small biases."""
    g = _generator(seed)
    x = torch.empty(case["n"], case["c"], case["h"], case["w"], device="cuda").uniform_(-1, 1, generator=g)
    std = math.sqrt(2.0 / (case["c"] * case["k"] ** 2))
    w = torch.empty(case["o"], case["c"], case["k"], case["k"], device="cuda").normal_(0, std, generator=g)
    b = torch.empty(case["o"], device="cuda").normal_(0, 0.01, generator=g)
    return g, x, w, b


_streams = []


def _compiled(func, case, x):
    """What a program that runs a graph keeps: the plan, the output buffer, and the one stream (not the default one, so that
    it can replay graphs) on which all its calls follow one another."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    graph = plan.CompiledGraph(func, precision=case["precision"], cuda_graph=True)
    out = torch.empty(graph.out_shape, device="cuda")
    return dict(graph=graph, stream=_streams[0], x=x, out=out)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        weights = resnet18.make_weights(seed)
        func = resnet18.build(case["n"], weights, to_constant=lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda())
        x = torch.empty(case["n"], 3, 224, 224, device="cuda").normal_(generator=_generator(seed))
        return dict(_compiled(func, case, x), kind="graph")
    if kind == "layer":
        _, x, w, b = _conv_tensors(case, seed)
        v = relay.Var("input", tuple(x.shape))
        p = case["k"] // 2
        attrs = relay.Conv2DAttrs((case["s"], case["s"]), (p, p, p, p), (1, 1), 1)
        conv = relay.Call("nn_conv2d", [v, relay.Constant(w), relay.Constant(b)], attrs)
        return dict(_compiled(relay.Function([v], relay.Call("nn_relu", [conv])), case, x), kind="graph")
    if kind == "conv":
        g, x, w, b = _conv_tensors(case, seed)
        r = torch.empty(case["n"], case["o"], *_out_hw(case), device="cuda").uniform_(-1, 1, generator=g)
        return dict(kind=kind, x=x, w=w, b=b, r=r, s=(case["s"],) * 2, p=(case["k"] // 2,) * 2, precision=case["precision"])
    if kind == "conv_s8":
        g = _generator(seed)
        n, c, h, w, o, k = (case[d] for d in ("n", "c", "h", "w", "o", "k"))
        xs, ws = ((n, h, w, c), (o, k, k, c)) if case["nhwc"] else ((n, c, h, w), (o, c, k, k))
        x = torch.randint(-128, 128, xs, device="cuda", generator=g, dtype=torch.int8)
        wt = torch.randint(-127, 128, ws, device="cuda", generator=g, dtype=torch.int8)
        b = torch.randint(-1000, 1001, (o,), device="cuda", generator=g, dtype=torch.int32)
        # multipliers in [2^30, 2^31), shifts that bring a sum of c*k*k products (rms 74 * 73 each) to int8
        m = torch.randint(1 << 30, (1 << 31) - 1, (o,), device="cuda", generator=g, dtype=torch.int64).to(torch.int32)
        bits = int(round(math.log2(5400.0 * math.sqrt(c * k * k) / 48.0)))
        sh = torch.randint(bits - 1, bits + 2, (o,), device="cuda", generator=g, dtype=torch.int32)
        return dict(kind=kind, x=x, w=wt, b=b, m=m, sh=sh, s=(case["s"],) * 2, p=(k // 2,) * 2, nhwc=case["nhwc"])
    if kind == "chain":
        g = _generator(seed)
        n, c, h, w = (case[d] for d in ("n", "c", "h", "w"))
        x = torch.empty(n, c, h, w, device="cuda").uniform_(-1, 1, generator=g)
        r = torch.empty(n, c, (h - 1) // 2 + 1, (w - 1) // 2 + 1, device="cuda").uniform_(-1, 1, generator=g)
        return dict(kind=kind, x=x, r=r)
    g = _generator(seed)
    x = torch.empty(case["n"], case["c"], case["h"], case["w"], device="cuda").uniform_(0, 2, generator=g)
    w = torch.empty(case["o"], case["c"], device="cuda").normal_(0, math.sqrt(2.0 / case["c"]), generator=g)
    b = torch.empty(case["o"], device="cuda").normal_(0, 0.01, generator=g)
    return dict(kind="head", x=x, w=w, b=b, precision=case["precision"])


def run(state):
    kind = state["kind"]
    if kind == "graph":
        with torch.cuda.stream(state["stream"]):
            return state["graph"].run(state["x"], out=state["out"])
    if kind == "conv":
        return ops.nn_conv2d(state["x"], state["w"], state["b"], strides=state["s"], padding=state["p"], residual=state["r"],
                             relu=True, precision=state["precision"])
    if kind == "conv_s8":
        return ops.nn_conv2d_s8(state["x"], state["w"], state["b"], state["m"], state["sh"], strides=state["s"],
                                padding=state["p"], relu=True, nhwc=state["nhwc"])
    if kind == "chain":
        return ops.max_pool2d_add_relu(state["x"], state["r"], (3, 3), (2, 2), (1, 1, 1, 1))
    y = ops.nn_flatten(ops.nn_global_avg_pool2d(state["x"]))
    return ops.softmax(ops.nn_gemm(y, state["w"], state["b"], transB=1, precision=state["precision"]))


def work(case):
    """Bytes of the inputs and weights as the caller hands them over and of the result; operations of the contractions.
    Intermediate activations of a network are not counted: they need not leave the chip."""
    kind = case["kind"]
    if kind == "net":
        n = case["n"]
        weights = 11_684_712 * 4.0  # 20 convolutions with their folded batch norms, and the classifier
        return {"bytes": n * (3 * 224 * 224 + 1000) * 4.0 + weights,
                "flops": float(n) * (resnet18.conv_flops_per_image() + resnet18.FC_FLOPS_PER_IMAGE)}
    if kind == "chain":
        n, c, h, w = (case[d] for d in ("n", "c", "h", "w"))
        out = n * c * ((h - 1) // 2 + 1) * ((w - 1) // 2 + 1)
        return {"bytes": 4.0 * (n * c * h * w + 2 * out), "flops": 11.0 * out}
    if kind == "head":
        n, c, o = case["n"], case["c"], case["o"]
        return {"bytes": 4.0 * (n * c * case["h"] * case["w"] + c * o + o + n * o), "flops": 2.0 * n * c * o}
    oh, ow = _out_hw(case)
    out = case["n"] * case["o"] * oh * ow
    elements = case["n"] * case["c"] * case["h"] * case["w"] + case["o"] * case["c"] * case["k"] ** 2
    if kind == "conv_s8":
        return {"bytes": float(elements + out + 12 * case["o"]), "flops": _conv_flops(case)}
    return {"bytes": 4.0 * (elements + case["o"] + out * (2 if kind == "conv" else 1)), "flops": _conv_flops(case)}


def tolerance(case):
    """Integers and the bit-exact float32 mode are equal. A bf16 network rounds every activation to 8 bits; tf32 rounds the
    operands of every contraction to 11; three passes leave the tensor core's own accumulation."""
    if case["kind"] in ("conv_s8", "chain") or case["precision"] == "fp32":
        return "exact"
    return {"rel": {"bf16": 1e-2, "tf32": 2e-3, "tf32x3": 1e-3}[case["precision"]]}
