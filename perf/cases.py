"""Workloads the forward path is timed on, through its public entry points.

Five kinds: a fully connected layer (``ip``), the GEMM interface (``gemm``), a convolution (``conv``), a depthwise-separable
block (``block``) and the whole ResNet-50 inference network (``net``).  Every input is made on the GPU from a seed: activations
~ N(0, 1), or that rectified where a layer follows a ReLU; weights Kaiming-normal; biases ~ U(-0.1, 0.1).  All data is fp32, the
only type of the path, which is forward only.
"""
import math

import numpy as np
import torch

from dlprimitives_b200 import capi, hostapi, resnet50

NET_SEED = 0            # the network's weights are the program's, not the request's: one set for all inputs
_net_params = {}
_service = {}           # the stream the program runs its networks on


def listed():
    return [
        # one request through a ResNet-50 classifier head whose weights were packed at start-up: the smallest call, all latency
        dict(name="ip_b1", kind="ip", batch=1, inputs=2048, outputs=1000, packed=True, act="identity"),
        # the same head on a full batch, weights as the interface takes them (packed on every call)
        dict(name="ip_b256_raw", kind="ip", batch=256, inputs=2048, outputs=1000, packed=False, act="identity"),
        # the GEMM interface on a large square product, C = A * B^T
        dict(name="gemm_2048", kind="gemm", batch=1, m=2048, n=2048, k=2048, ta=False, tb=True, bias=0, act="identity"),
        # a batch of ragged products with both operands the other way round
        dict(name="gemm_ragged_batch5", kind="gemm", batch=5, m=333, n=517, k=1001, ta=True, tb=False, bias=0, act="identity"),
        # a single 3x3 layer at a moderate batch, bias and ReLU fused, weights passed on every call
        dict(name="conv3x3_64_56_n16", kind="conv", batch=16, cin=64, cout=64, hw=56, k=3, stride=1, pad=1, act="relu", packed=False,
             res=False, relu_in=False, algo=""),
        # a bottleneck's 1x1 expansion with its residual sum fused, weights packed
        dict(name="conv1x1_256_1024_14_n64", kind="conv", batch=64, cin=256, cout=1024, hw=14, k=1, stride=1, pad=0, act="identity",
             packed=True, res=True, relu_in=True, algo=""),
        # a wide kernel on an odd plane (AlexNet's second layer)
        dict(name="conv5x5_64_192_27_n64", kind="conv", batch=64, cin=64, cout=192, hw=27, k=5, stride=1, pad=2, act="relu", packed=True,
             res=False, relu_in=True, algo=""),
        # the Winograd algorithm, on request
        dict(name="winograd_256_14_n64", kind="conv", batch=64, cin=256, cout=256, hw=14, k=3, stride=1, pad=1, act="relu", packed=True,
             res=False, relu_in=True, algo="winograd"),
        # a MobileNetV2 row: depthwise 3x3, then the 1x1 projection with ReLU6
        dict(name="block_144_24_56_n128", kind="block", batch=128, c=144, cout=24, hw=56, stride=1),
        # the network for one image at a time (a service without batching)
        dict(name="resnet50_b1", kind="net", batch=1, size=224, folded=True),
        # the form the reference ships (BatchNorm and ReLU as operators of their own) at the batch of its benchmark file
        dict(name="resnet50_bn_b16", kind="net", batch=16, size=224, folded=False),
        # the headline workload: whole batches of 256
        dict(name="resnet50_b256", kind="net", batch=256, size=224, folded=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ip", "gemm", "conv", "conv", "conv", "conv", "block", "net"])
    if kind == "ip":
        return dict(kind=kind, batch=_log_int(rng, 1, 1024), inputs=_log_int(rng, 256, 9216), outputs=_log_int(rng, 10, 4096),
                    packed=rng.random() < 0.5, act=rng.choice(["identity", "relu"]))
    if kind == "gemm":
        batch = rng.choice([1, 1, 1, 4, 8])
        top = 4096 if batch == 1 else 1024
        return dict(kind=kind, batch=batch, m=_log_int(rng, 64, top), n=_log_int(rng, 64, top), k=_log_int(rng, 64, top),
                    ta=rng.random() < 0.3, tb=rng.random() < 0.6, bias=rng.choice([0, 2]) if batch == 1 else 0,
                    act=rng.choice(["identity", "relu"]) if batch == 1 else "identity")
    if kind == "block":
        hw = rng.choice([112, 56, 28, 14, 7, _log_int(rng, 9, 120)])
        c = 8 * _log_int(rng, 4, 120)
        batch = max(1, min(_log_int(rng, 8, 128), int(4e8 // (c * hw * hw))))
        return dict(kind=kind, batch=batch, c=c, cout=8 * _log_int(rng, 2, 40), hw=hw, stride=rng.choice([1, 2]))
    if kind == "net":
        return dict(kind=kind, batch=_log_int(rng, 1, 128), size=rng.choice([224, 224, 192, 160, 225, _log_int(rng, 128, 256)]),
                    folded=rng.random() < 0.75)
    k = rng.choice([1, 1, 3, 3, 3, 5, 7])
    hw = _log_int(rng, 7, 112)
    if k == 7:
        cin, cout, stride, hw = rng.choice([1, 3, 4]), rng.choice([32, 64, 96]), 2, _log_int(rng, 64, 256)
    else:
        # channel counts: mostly the powers of two of the benchmark networks, or anything
        cin = rng.choice([64, 128, 256, 512, 1024 if k == 1 else 192, _log_int(rng, 16, 512)])
        cout = rng.choice([64, 128, 256, 512, 2048 if k == 1 else 384, _log_int(rng, 16, 512)])
        stride = rng.choice([1, 1, 1, 2])
    flops1 = 2.0 * cin * cout * k * k * (hw // stride + 1) ** 2
    bytes1 = 4.0 * (cin * hw * hw + 2 * cout * (hw // stride + 1) ** 2)
    batch = max(1, min(_log_int(rng, 1, 256), int(2e11 / flops1), int(2e9 / bytes1)))
    return dict(kind=kind, batch=batch, cin=cin, cout=cout, hw=hw, k=k, stride=stride, pad=k // 2, act=rng.choice(["identity", "relu", "relu6"]),
                packed=rng.random() < 0.7, res=k == 1 and stride == 1 and rng.random() < 0.4, relu_in=rng.random() < 0.6,
                algo="winograd" if k == 3 and stride == 1 and rng.random() < 0.2 else "")


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0, relu=False):
    t = torch.randn(*shape, device="cuda", generator=g)
    if relu:
        t.relu_()
    return t.mul_(std) if std != 1.0 else t


def _uniform(g, n):
    return torch.rand(n, device="cuda", generator=g).mul_(0.2).sub_(0.1)


def _bytes(n):
    return torch.empty(max(int(n), 16), dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "ip":
        b, i, o = case["batch"], case["inputs"], case["outputs"]
        plan = capi.IPForward(i, o, b, bias=True, activation=case["act"])
        s = dict(kind=kind, plan=plan, x=_randn(g, b, i, relu=True), w=_randn(g, o, i, std=math.sqrt(2.0 / i)), bias=_uniform(g, o),
                 y=torch.empty(b, o, device="cuda"), ws=_bytes(plan.workspace()), packed=None)
        if case["packed"]:
            s["packed"] = plan.prepack(s["w"])
        return s
    if kind == "gemm":
        m, n, k, cnt = case["m"], case["n"], case["k"], case["batch"]
        plan = capi.Gemm(case["ta"], case["tb"], m, n, k, bias_mode=case["bias"], activation=case["act"])
        a = _randn(g, *([cnt] if cnt > 1 else []), *((k, m) if case["ta"] else (m, k)))
        b = _randn(g, *([cnt] if cnt > 1 else []), *((n, k) if case["tb"] else (k, n)))
        ws = _bytes(plan.batched_workspace(cnt) if cnt > 1 else plan.workspace())
        return dict(kind=kind, plan=plan, cnt=cnt, m=m, n=n, k=k, a=a, lda=m if case["ta"] else k, b=b, ldb=k if case["tb"] else n,
                    bias=_uniform(g, n) if case["bias"] else None, c=torch.empty(cnt, m, n, device="cuda"), ws=ws)
    if kind == "conv":
        b, cin, cout, hw, k = case["batch"], case["cin"], case["cout"], case["hw"], case["k"]
        plan = capi.Conv2DForward(channels_in=cin, channels_out=cout, kernel=k, stride=case["stride"], pad=case["pad"], batch=b, height=hw,
                                  width=hw, bias=True, activation=case["act"], algo=case["algo"])
        shape = plan.output_shape(b)
        s = dict(kind=kind, plan=plan, x=_randn(g, b, cin, hw, hw, relu=case["relu_in"]),
                 w=_randn(g, cout, cin, k, k, std=math.sqrt(2.0 / (cin * k * k))), bias=_uniform(g, cout), y=torch.empty(shape, device="cuda"),
                 ws=_bytes(plan.workspace()), packed=None, res=_randn(g, *shape) if case["res"] else None)
        if case["packed"] or case["res"]:
            s["packed"] = plan.prepack(s["w"])
        return s
    if kind == "block":
        b, c, hw = case["batch"], case["c"], case["hw"]
        dw = hostapi.Operator("Convolution2D", {"channels_in": c, "channels_out": c, "kernel": 3, "pad": 1, "stride": case["stride"],
                                                "groups": c, "bias": True, "activation": "relu6"}, [(b, c, hw, hw)])
        mid = dw.out_shapes[0]
        pw = hostapi.Operator("Convolution2D", {"channels_in": c, "channels_out": case["cout"], "kernel": 1, "bias": True,
                                                "activation": "relu6"}, [mid])
        return dict(kind=kind, dw=dw, pw=pw, x=_randn(g, b, c, hw, hw, relu=True).clamp_(max=6.0),
                    dw_params=[_randn(g, c, 1, 3, 3, std=math.sqrt(2.0 / 9)), _uniform(g, c)],
                    pw_params=[_randn(g, case["cout"], c, 1, 1, std=math.sqrt(2.0 / c)), _uniform(g, case["cout"])],
                    mid=torch.empty(mid, device="cuda"), y=torch.empty(pw.out_shapes[0], device="cuda"))
    # the network: built, its weights uploaded; the service hands it one device tensor per request, on its own stream
    net_json = _net_json(case)
    if case["folded"] not in _net_params:
        # random weights let the activations grow through the residual sums; the classifier is scaled so that its logits have a
        # trained network's spread (standard deviation about 2) and the softmax is not a one
        params = resnet50.make_params(net_json, seed=NET_SEED)
        params["fc.0"] = params["fc.0"] * np.float32(1.0 / 2000)
        _net_params[case["folded"]] = params
    net = hostapi.Net(net_json)
    for name, value in _net_params[case["folded"]].items():
        net.set_param(name, value)
    net.upload_params()
    if "stream" not in _service:
        _service["stream"] = torch.cuda.Stream()
    return dict(kind="net", net=net, x=_randn(g, case["batch"], 3, case["size"], case["size"]), stream=_service["stream"],
                fc=torch.empty(case["batch"], 1000, device="cuda"), prob=torch.empty(case["batch"], 1000, device="cuda"))


def _net_json(case):
    net_json = resnet50.make_json(case["batch"], case["size"], case["size"], folded=case["folded"])
    net_json["outputs"] = ["fc", "prob"]
    return net_json


def run(s):
    kind = s["kind"]
    if kind == "ip":
        if s["packed"] is None:
            s["plan"].enqueue(s["x"], s["w"], s["bias"], s["y"], ws=s["ws"])
        else:
            s["plan"].enqueue_packed(s["x"], s["packed"], s["bias"], s["y"], ws=s["ws"])
        return s["y"]
    if kind == "gemm":
        m, n, k = s["m"], s["n"], s["k"]
        if s["cnt"] > 1:
            s["plan"].batch_gemm(s["cnt"], m, n, k, s["a"], m * k, s["lda"], s["b"], n * k, s["ldb"], s["c"], m * n, n, ws=s["ws"])
        else:
            s["plan"].gemm(m, n, k, s["a"], s["lda"], s["b"], s["ldb"], s["c"], n, bias=s["bias"], ws=s["ws"])
        return s["c"]
    if kind == "conv":
        if s["packed"] is None:
            s["plan"].enqueue(s["x"], s["w"], s["bias"], s["y"], ws=s["ws"])
        elif s["res"] is None:
            s["plan"].enqueue_packed(s["x"], s["packed"], s["bias"], s["y"], ws=s["ws"])
        else:
            s["plan"].enqueue_packed(s["x"], s["packed"], s["bias"], s["y"], residual=s["res"], post_activation="relu", ws=s["ws"])
        return s["y"]
    if kind == "block":
        s["dw"].forward([s["x"]], s["dw_params"], [s["mid"]])
        s["pw"].forward([s["mid"]], s["pw_params"], [s["y"]])
        return s["y"]
    net, stream = s["net"], s["stream"]
    net.copy_tensor_from("data", s["x"], stream)
    net.forward(stream)
    net.copy_tensor_to("fc", s["fc"], stream)
    net.copy_tensor_to("prob", s["prob"], stream)
    return {"fc": s["fc"], "prob": s["prob"]}


def work(case):
    kind = case["kind"]
    if kind == "ip":
        b, i, o = case["batch"], case["inputs"], case["outputs"]
        return {"bytes": 4.0 * (b * i + i * o + o + b * o), "flops": 2.0 * b * i * o}
    if kind == "gemm":
        m, n, k, cnt = case["m"], case["n"], case["k"], case["batch"]
        return {"bytes": 4.0 * cnt * (m * k + k * n + m * n), "flops": 2.0 * cnt * m * n * k}
    if kind == "conv":
        out = (case["hw"] + 2 * case["pad"] - case["k"]) // case["stride"] + 1
        y = float(case["batch"]) * case["cout"] * out * out
        x = float(case["batch"]) * case["cin"] * case["hw"] ** 2
        w = float(case["cin"]) * case["cout"] * case["k"] ** 2
        return {"bytes": 4.0 * (x + y * (2 if case["res"] else 1) + w + case["cout"]), "flops": 2.0 * y * case["cin"] * case["k"] ** 2}
    if kind == "block":
        out = (case["hw"] - 1) // case["stride"] + 1
        x = float(case["batch"]) * case["c"] * case["hw"] ** 2
        mid = float(case["batch"]) * case["c"] * out * out
        y = float(case["batch"]) * case["cout"] * out * out
        # the two operators are two calls: the tensor between them is an output of one and an input of the other
        return {"bytes": 4.0 * (x + 2 * mid + y + case["c"] * (9 + case["cout"])), "flops": 18.0 * mid + 2.0 * y * case["c"]}
    net_json = _net_json(case)
    weights = 25.5e6
    return {"bytes": 4.0 * (case["batch"] * (3.0 * case["size"] ** 2 + 2000) + weights), "flops": float(case["batch"]) * resnet50.flops_per_image(net_json)}


def tolerance(case):
    # About four times what the path differs by from itself in 64 bits: single calls rel 2.2e-6, max 1.0e-5; the network's 54
    # layers carry each other's rounding on: logits (spread 2) rel 5.0e-5, and the probabilities by as much as the logits differ, 1e-4.
    if case["kind"] == "net":
        return {"rel": 4e-4, "max": 1.6e-3}
    return {"rel": 1e-5, "max": 5e-5}


# ---- the same results in 64 bits, with plain torch ----------------------------------------------------------------------

def _act64(y, act):
    return y.clamp_(min=0.0) if act == "relu" else (y.clamp_(0.0, 6.0) if act == "relu6" else y)


def _conv64(x, w, bias, stride, pad, act="identity"):
    """A dense convolution as patches times weights, a few images at a time."""
    n, _, h, wd = x.shape
    o, _, kh, kw = w.shape
    oh, ow = (h + 2 * pad - kh) // stride + 1, (wd + 2 * pad - kw) // stride + 1
    w64 = w.double().reshape(o, -1)
    y = torch.empty(n, o, oh, ow, dtype=torch.float64, device=x.device)
    step = max(1, int(2e8 // (w64.shape[1] * oh * ow)))
    for i in range(0, n, step):
        part = x[i:i + step].double()
        if kh == kw == 1:
            cols = part[:, :, ::stride, ::stride].reshape(part.shape[0], part.shape[1], -1)
        else:
            cols = torch.nn.functional.unfold(part, (kh, kw), padding=pad, stride=stride)
        r = torch.matmul(w64, cols)
        if bias is not None:
            r += bias.double()[:, None]
        y[i:i + step] = _act64(r, act).reshape(part.shape[0], o, oh, ow)
    return y


def _depthwise64(x, w, bias, stride, act):
    n, c, h, wd = x.shape
    oh, ow = (h - 1) // stride + 1, (wd - 1) // stride + 1
    xp = torch.nn.functional.pad(x.double(), (1, 1, 1, 1))
    y = bias.double()[None, :, None, None].expand(n, c, oh, ow).clone()
    for i in range(3):
        for j in range(3):
            y += w[:, 0, i, j].double()[None, :, None, None] * xp[:, :, i:i + (oh - 1) * stride + 1:stride, j:j + (ow - 1) * stride + 1:stride]
    return _act64(y, act)


def _net64(net_json, params, x):
    """The network's operators one by one; every parameter and the input are the fp32 values the network has."""
    p = {name: torch.from_numpy(value).to(x.device) for name, value in params.items()}
    t = {net_json["inputs"][0]["name"]: x.double()}
    last = {name: i for i, op in enumerate(net_json["operators"]) for name in op["inputs"]}
    for i, op in enumerate(net_json["operators"]):
        o, src, name = op["options"], [t[k] for k in op["inputs"]], op["name"]
        if op["type"] == "Convolution2D":
            y = _conv64(src[0], p[name + ".0"], p.get(name + ".1") if o["bias"] else None, o["stride"][0], o["pad"][0], o.get("activation", "identity"))
        elif op["type"] == "BatchNorm":
            mean, var, gamma, beta = [p["%s.%d" % (name, k)].double()[None, :, None, None] for k in range(4)]
            y = (src[0] - mean) / (var + o["eps"]).sqrt() * gamma + beta
        elif op["type"] == "Activation":
            y = _act64(src[0].clone(), o["activation"])
        elif op["type"] == "Pooling2D":
            y = torch.nn.functional.max_pool2d(src[0], o["kernel"], o["stride"], o["pad"])
        elif op["type"] == "Elementwise":
            y = _act64(src[0] + src[1], o["activation"])
        elif op["type"] == "GlobalPooling":
            y = src[0].mean(dim=(2, 3))
        elif op["type"] == "InnerProduct":
            y = src[0] @ p[name + ".0"].double().t() + p[name + ".1"].double()
        else:
            y = torch.softmax(src[0], dim=1)
        t[op["outputs"][0]] = y
        for k in op["inputs"]:
            if last[k] == i and k not in net_json["outputs"]:
                t.pop(k, None)
    return t


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "ip":
        return _act64(s["x"].double() @ s["w"].double().t() + s["bias"].double(), case["act"])
    if kind == "gemm":
        a, b = s["a"].double(), s["b"].double()
        c = (a.transpose(-1, -2) if case["ta"] else a) @ (b.transpose(-1, -2) if case["tb"] else b)
        if s["bias"] is not None:
            c = c + s["bias"].double()
        return _act64(c, case["act"]).reshape(s["c"].shape)
    if kind == "conv":
        y = _conv64(s["x"], s["w"], s["bias"], case["stride"], case["pad"], case["act"])
        return torch.relu_(y.add_(s["res"])) if case["res"] else y
    if kind == "block":
        mid = _depthwise64(s["x"], s["dw_params"][0], s["dw_params"][1], case["stride"], "relu6")
        return _conv64(mid, s["pw_params"][0], s["pw_params"][1], 1, 0, "relu6")
    net_json = _net_json(case)
    fc, prob, step = [], [], 32
    for i in range(0, case["batch"], step):
        t = _net64(net_json, _net_params[case["folded"]], s["x"][i:i + step])
        fc.append(t["fc"])
        prob.append(t["prob"])
    return {"fc": torch.cat(fc), "prob": torch.cat(prob)}
