"""The workloads that the performance of this library is followed on.

Each case is work a program has the library do through its public Python entry points
(portdnn_b200.api and the layer-table runner of portdnn_b200.workloads): whole networks, forward and
training, from one image to the benchmark batch; single layers of odd sizes in all three passes; and the
operators around the convolutions in the sequences a network runs them in.  ``listed()`` names the ones
that are followed, ``draw()`` gives further ones of the same ranges.
"""
import math

import torch

from portdnn_b200 import api, workloads

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
CODES = {"f16": api.F16, "bf16": api.BF16, "f32": api.F32}


def listed():
    return [
        # one image through a network: the answer to a single request, where latency is what counts
        {"name": "resnet50_forward_b1", "kind": "net", "net": "resnet50", "mode": "forward", "batch": 1, "dtype": "f16"},
        # the benchmark configuration of the library: offline inference at full batch
        {"name": "resnet50_forward_b256", "kind": "net", "net": "resnet50", "mode": "forward", "batch": 256, "dtype": "f16"},
        # the backward pass of a training step with a small share of the batch per GPU, as in fine-tuning
        {"name": "resnet50_backward_b24", "kind": "net", "net": "resnet50", "mode": "backward", "batch": 24, "dtype": "bf16"},
        # the backward pass of the training benchmark: one GPU's share of a global batch of 2048
        {"name": "resnet50_backward_b256", "kind": "net", "net": "resnet50", "mode": "backward", "batch": 256, "dtype": "f16"},
        # a whole training step in single precision (3xTF32), on a network of 3x3 layers only
        {"name": "vgg16_train_f32_b8", "kind": "net", "net": "vgg16", "mode": "train", "batch": 8, "dtype": "f32"},
        # depthwise-separable network: short HBM-bound layers, depthwise kernels, activations, residual adds
        {"name": "mobilenet_forward_b64", "kind": "mobilenet", "batch": 64, "dtype": "f16"},
        # a depthwise layer in training, all three passes
        {"name": "depthwise_train_56x56x144", "kind": "depthwise", "batch": 128, "rows": 56, "cols": 56, "channels": 144,
         "window": 3, "stride": 1, "dtype": "f16"},
        # a layer of a pruned network on a cropped image: nothing is a multiple of anything; all three passes
        {"name": "conv_ragged_train", "kind": "conv", "batch": 7, "rows": 45, "cols": 61, "channels": 100, "features": 150,
         "window": 3, "stride": 1, "dtype": "bf16"},
        # convolution, batch normalisation and ReLU in training, forward and backward
        {"name": "conv_bn_relu_train", "kind": "norm", "batch": 64, "rows": 28, "cols": 28, "channels": 128, "features": 256,
         "window": 1, "dtype": "f16"},
        # grouped 3x3 convolution of a wide bottleneck
        {"name": "grouped_conv_forward", "kind": "grouped", "batch": 32, "rows": 28, "cols": 28, "channels": 512,
         "features": 512, "groups": 32, "window": 3, "stride": 1, "dtype": "f16"},
        # the end of a classifier: global average pool, fully connected layer, bias, softmax, and their gradients
        {"name": "classifier_head_train", "kind": "head", "batch": 250, "size": 7, "channels": 2048, "classes": 1000,
         "dtype": "f16"},
        # 3x3/2 and 2x2/2 max pooling with their gradients on an odd-sized image
        {"name": "pool_train_f32", "kind": "pool", "batch": 16, "rows": 113, "cols": 151, "channels": 64, "dtype": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kind first, then its sizes over the logarithm of their range."""
    kind = rng.choice(["resnet50", "resnet50_backward", "vgg16", "mobilenet", "depthwise", "conv", "conv", "norm", "grouped",
                       "head", "pool"])
    half = rng.choice(["f16", "bf16"])
    if kind == "resnet50":
        return {"kind": "net", "net": "resnet50", "mode": "forward", "batch": _log(rng, 1, 256), "dtype": half}
    if kind == "resnet50_backward":
        return {"kind": "net", "net": "resnet50", "mode": "backward", "batch": _log(rng, 4, 192), "dtype": half}
    if kind == "vgg16":
        dtype, mode = rng.choice([("f32", "forward"), ("f32", "train"), ("f16", "forward"), ("f16", "backward")])
        return {"kind": "net", "net": "vgg16", "mode": mode, "batch": _log(rng, 1, 10), "dtype": dtype}
    if kind == "mobilenet":
        return {"kind": "mobilenet", "batch": _log(rng, 1, 160), "dtype": "f16"}
    if kind == "depthwise":
        rows, channels, stride = _log(rng, 7, 120), 8 * _log(rng, 3, 120), rng.choice([1, 1, 2])
        cols = max(7, min(160, rows + rng.randint(-6, 20)))
        most = max(1, int(6e7 / (rows * cols * channels)))
        return {"kind": "depthwise", "batch": _log(rng, 1, min(128, most)), "rows": rows, "cols": cols, "channels": channels,
                "window": 3, "stride": stride, "dtype": half}
    if kind == "conv":
        rows, window, stride = _log(rng, 7, 90), rng.choice([1, 3, 3, 5]), rng.choice([1, 1, 2])
        cols = max(7, rows + rng.randint(-5, 25))
        channels, features = _log(rng, 12, 520), _log(rng, 12, 520)
        if rng.random() < 0.4:  # widths as networks mostly have them
            channels, features = (channels + 15) // 16 * 16, (features + 15) // 16 * 16
        per_image = 2.0 * rows * cols * channels * features * window * window / stride ** 2
        return {"kind": "conv", "batch": _log(rng, 1, max(1, min(64, int(1.2e10 / per_image)))), "rows": rows, "cols": cols,
                "channels": channels, "features": features, "window": window, "stride": stride,
                "dtype": rng.choice(["f16", "bf16", "bf16", "f32"])}
    if kind == "norm":
        rows, channels, features = _log(rng, 7, 80), 8 * _log(rng, 4, 64), 8 * _log(rng, 4, 128)
        cols = max(7, rows + rng.randint(-4, 12))
        most = max(1, int(8e7 / (rows * cols * max(channels, features))))
        return {"kind": "norm", "batch": _log(rng, 1, min(128, most)), "rows": rows, "cols": cols, "channels": channels,
                "features": features, "window": rng.choice([1, 1, 3]), "dtype": half}
    if kind == "grouped":
        size, groups, width = _log(rng, 7, 60), rng.choice([2, 4, 8, 16, 32, 32, 64]), 8 * rng.randint(1, 4)
        most = max(1, int(3e7 / (size * size * groups * width)))
        return {"kind": "grouped", "batch": _log(rng, 1, min(64, most)), "rows": size, "cols": size + rng.randint(0, 3),
                "channels": groups * width, "features": groups * width, "groups": groups, "window": 3,
                "stride": rng.choice([1, 1, 2]), "dtype": half}
    if kind == "head":
        return {"kind": "head", "batch": _log(rng, 1, 512), "size": rng.randint(5, 9), "channels": 8 * _log(rng, 16, 256),
                "classes": _log(rng, 10, 1100), "dtype": rng.choice(["f16", "bf16", "f32"])}
    rows, channels = _log(rng, 14, 230), 4 * _log(rng, 2, 64)
    cols = max(14, rows + rng.randint(-10, 40))
    most = max(1, int(6e7 / (rows * cols * channels)))
    return {"kind": "pool", "batch": _log(rng, 1, min(128, most)), "rows": rows, "cols": cols, "channels": channels,
            "dtype": rng.choice(["f32", "f16", "bf16"])}


# ---- whole networks from the layer tables --------------------------------------------------------


def _layers(case):
    return {"resnet50": workloads.resnet50_v15, "vgg16": workloads.vgg16}[case["net"]](case["batch"])


def _prepare_net(case, seed):
    dt = DTYPES[case["dtype"]]
    r = workloads.ConvStackRunner(_layers(case), torch.device("cuda"), seed, training=case["mode"] != "forward", dtype=dt)
    if case["mode"] == "backward":
        _fill_activations(r, torch.Generator(device="cuda").manual_seed(seed + 1000003), dt)
    return {"runner": r, "mode": case["mode"]}


def _fill_activations(r, g, dt):
    """What a forward pass leaves for the backward pass: the output of every layer - with He-normal weights a
    rectified normal - and the sign bits of those that are kept as bits.  Drawn instead of computed: a
    16-bit forward pass that rounds one value differently flips ReLU masks further on, and gradients behind
    tens of masks then have a fifth of their norm in common masks only, whichever of the two is looked at."""
    one = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device="cuda")
    for i, l in enumerate(r.layers):
        if isinstance(l, workloads.ConvLayer):
            torch.randn(r.sizes[i], device="cuda", generator=g, dtype=dt, out=r.acts[i])
            if l.activation == api.ACT_RELU:
                r.acts[i].relu_()
        elif r.src_idx[i] >= 0 and l.op == api.POOL_MAX:
            p = l.params
            x = r.acts[r.src_idx[i]].view(p.batch, p.in_rows, p.in_cols, p.channels).permute(0, 3, 1, 2)
            below, right = ((o - 1) * s + w - n - pad for o, s, w, n, pad in (
                (p.out_rows, p.stride_rows, p.window_rows, p.in_rows, p.pad_rows),
                (p.out_cols, p.stride_cols, p.window_cols, p.in_cols, p.pad_cols)))
            x = torch.nn.functional.pad(x, (p.pad_cols, max(right, 0), p.pad_rows, max(below, 0)))  # (no input is negative)
            y = torch.nn.functional.max_pool2d(x, p.window_rows, p.stride_rows)
            r.acts[i].copy_(y.permute(0, 2, 3, 1).reshape(-1))
        if i in r.bits:
            r.bits[i].copy_(((r.acts[i].view(-1, 8) > 0) * one).sum(1, dtype=torch.uint8))


def _run_net(s):
    r = s["runner"]
    if s["mode"] == "forward":
        return r.forward()
    if s["mode"] == "backward":
        r.backward()
        return {"filter_gradients": [r.bucket.view(k) for k in range(len(r.conv_ids))]}
    r.train_step()
    return {"output": r.acts[-1], "filter_gradients": [r.bucket.view(k) for k in range(len(r.conv_ids))]}


def _work_net(case):
    es = 4 if case["dtype"] == "f32" else 2
    forward, backward = case["mode"] != "backward", case["mode"] != "forward"
    flops, moved = 0, 0
    for l in _layers(case):
        p = l.params
        if isinstance(l, workloads.PoolLayer):
            io = es * p.batch * p.channels * (p.in_rows * p.in_cols + p.out_rows * p.out_cols)
            moved += io * forward
            if backward and l.op == api.POOL_MAX and p.in_rows > 14:  # (the last pool's gradient is not asked for)
                moved += 2 * io  # both sides and the gradient read, the gradient written
            continue
        x, y = p.batch * p.in_rows * p.in_cols * p.channels, _conv_out(p)
        w = p.window_rows * p.window_cols * p.channels * p.features
        if forward:
            flops += l.flops
            moved += es * (x + w + y)
        if backward:
            first = l.src == "input"
            flops += l.flops * (1 if first else 2)
            moved += es * (x + y) + 4 * w + (0 if first else es * (y + w + x))
    return {"bytes": moved, "flops": flops}


# ---- MobileNet-v2 forward with its depthwise layers -----------------------------------------------


def _mobilenet_plan(batch):
    """(operator, its parameters, buffer read, buffer written): 3x3/2 stem, then per inverted-residual block
    the 1x1 expansion, the 3x3 depthwise layer with its ReLU6, the linear 1x1 projection and, where the
    shapes allow, the residual add."""
    convs, depth = iter(workloads.mobilenet_v2_convs(batch)), iter(workloads.mobilenet_v2_depthwise(batch))
    stem = next(convs)
    steps = [("conv", stem.params, api.ACT_RELU6)]
    for t, c, n, _ in ((1, 16, 1, 1), (6, 24, 2, 2), (6, 32, 3, 2), (6, 64, 4, 2), (6, 96, 3, 1), (6, 160, 3, 2), (6, 320, 1, 1)):
        for i in range(n):
            if t != 1:
                steps.append(("conv", next(convs).params, api.ACT_RELU6))
            steps.append(("depthwise", next(depth), None))
            steps.append(("relu6", None, None))
            steps.append(("conv", next(convs).params, api.ACT_NONE))
            if i > 0:
                steps.append(("add", None, None))
    return steps


def _conv_out(p):
    return p.batch * p.out_rows * p.out_cols * p.features


def _prepare_mobilenet(case, seed):
    dt, g = DTYPES[case["dtype"]], torch.Generator(device="cuda").manual_seed(seed)
    steps, biggest = [], 0
    for op, p, act in _mobilenet_plan(case["batch"]):
        st = {"op": op, "params": p, "act": act}
        if op == "conv":
            fan = p.window_rows * p.window_cols * p.channels
            # the linear projections at half He scale: in a trained network a residual branch is the smaller part
            scale = (2.0 / fan) ** 0.5 * (0.5 if act == api.ACT_NONE else 1.0)
            st["w"] = (torch.randn(fan * p.features, device="cuda", generator=g) * scale).to(dt)
            st["b"] = (torch.randn(p.features, device="cuda", generator=g) * 0.01).to(dt)
            _, rec = api.conv2d_workspace_size(api.FORWARD, CODES[case["dtype"]], p, api.ALGO_IM2COL)
            st["ws"] = torch.empty(rec, dtype=dt, device="cuda") if rec else None
            n = _conv_out(p)
        elif op == "depthwise":
            st["w"] = (torch.randn(9 * p.channels, device="cuda", generator=g) * 0.4).to(dt)
            n = p.batch * p.out_rows * p.out_cols * p.channels
        biggest = max(biggest, n)
        st["n"] = n
        steps.append(st)
    for st, after in zip(steps, steps[1:] + [{"op": None}]):
        st["ends_block"] = st["op"] == "add" or (st["op"] == "conv" and st["act"] == api.ACT_NONE and after["op"] != "add")
    x = torch.randn(case["batch"] * 224 * 224 * 3, device="cuda", generator=g).to(dt)
    buf = [torch.empty(biggest, dtype=dt, device="cuda") for _ in range(4)]
    return {"steps": steps, "x": x, "buf": buf}


def _run_mobilenet(s):
    buf, cur, block = s["buf"], s["x"], None  # block: the tensor a residual add comes back to
    where = -1
    for st in s["steps"]:
        op, n = st["op"], st["n"]
        if op == "add":
            cur = api.binaryop(api.BINARY_ADD, cur, [n], block, [n], out=cur)
        elif op == "relu6":
            cur = api.pointwise(api.ACT_RELU6, cur, out=cur)
        else:
            used = {where} | ({s["block_at"]} if block is not None else set())
            to = next(i for i in range(4) if i not in used)
            out = buf[to][:n]
            if op == "conv":
                cur = api.conv2d(api.FORWARD, cur, st["w"], st["params"], out=out, bias=st["b"], activation=st["act"],
                                 workspace=st["ws"], constant_filter=True)
            else:
                cur = api.depthwise_conv2d(api.FORWARD, cur, st["w"], st["params"], out=out)
            where = to
        if st["ends_block"]:
            block, s["block_at"] = cur, where
    return cur


def _work_mobilenet(case):
    flops, moved, n = 0, 0, 0
    for op, p, _ in _mobilenet_plan(case["batch"]):
        if op == "conv":
            n = _conv_out(p)
            w = p.window_rows * p.window_cols * p.channels * p.features
            flops += 2 * p.batch * p.out_rows * p.out_cols * w
            moved += 2 * (p.batch * p.in_rows * p.in_cols * p.channels + w + n)
        elif op == "depthwise":
            n = p.batch * p.out_rows * p.out_cols * p.channels
            flops += 18 * n
            moved += 2 * (p.batch * p.in_rows * p.in_cols * p.channels + 9 * p.channels + n)
        else:
            moved += 2 * n * (2 if op == "relu6" else 3)
    return {"bytes": moved, "flops": flops}


# ---- single layers in training ---------------------------------------------------------------------


def _randn(g, n, dt, scale=1.0):
    return (torch.randn(n, device="cuda", generator=g) * scale).to(dt)


def _depthwise_params(case):
    p = api.depthwise_params(case["batch"], case["rows"], case["cols"], case["channels"], 1, case["window"], case["stride"])
    return p, p.batch * p.in_rows * p.in_cols * p.channels, p.batch * p.out_rows * p.out_cols * p.channels


def _prepare_depthwise(case, seed):
    dt, g = DTYPES[case["dtype"]], torch.Generator(device="cuda").manual_seed(seed)
    p, nx, ny = _depthwise_params(case)
    taps = case["window"] ** 2
    ws = api.depthwise_workspace_bytes(api.FILTER_BACKPROP, CODES[case["dtype"]], p)
    return {"p": p, "x": _randn(g, nx, dt), "w": _randn(g, taps * p.channels, dt, (2.0 / taps) ** 0.5), "dy": _randn(g, ny, dt),
            "ws": torch.empty(max(ws, 16), dtype=torch.uint8, device="cuda")}


def _run_depthwise(s):
    y = api.depthwise_conv2d(api.FORWARD, s["x"], s["w"], s["p"])
    dw = api.depthwise_conv2d(api.FILTER_BACKPROP, s["x"], s["dy"], s["p"], workspace=s["ws"])
    dx = api.depthwise_conv2d(api.INPUT_BACKPROP, s["dy"], s["w"], s["p"])
    return {"y": y, "dw": dw, "dx": dx}


def _work_depthwise(case):
    p, nx, ny = _depthwise_params(case)
    taps = case["window"] ** 2
    return {"bytes": 2 * 3 * (nx + ny + taps * p.channels), "flops": 3 * 2 * taps * ny}


def _conv_params(case):
    return api.conv_params(case["batch"], case["rows"], case["cols"], case["channels"], case["features"], case["window"],
                           case.get("stride", 1), groups=case.get("groups", 1))


def _conv_sizes(p):
    return (p.batch * p.in_rows * p.in_cols * p.channels, p.window_rows * p.window_cols * p.channels // p.groups * p.features,
            _conv_out(p))


def _prepare_conv(case, seed):
    dt, g = DTYPES[case["dtype"]], torch.Generator(device="cuda").manual_seed(seed)
    p = _conv_params(case)
    nx, nw, ny = _conv_sizes(p)
    s = {"p": p, "x": _randn(g, nx, dt), "w": _randn(g, nw, dt, (2.0 * p.features / nw) ** 0.5),
         "b": _randn(g, p.features, dt, 0.01)}
    if p.groups == 1:
        s["dy"] = _randn(g, ny, dt)
        for key, which in (("ws", api.FORWARD), ("ws_dw", api.FILTER_BACKPROP)):
            _, rec = api.conv2d_workspace_size(which, CODES[case["dtype"]], p, api.ALGO_IM2COL)
            s[key] = torch.empty(rec, dtype=dt, device="cuda") if rec else None
    return s


def _run_conv(s):
    y = api.conv2d(api.FORWARD, s["x"], s["w"], s["p"], bias=s["b"], activation=api.ACT_RELU, workspace=s["ws"])
    dw = api.conv2d(api.FILTER_BACKPROP, s["x"], s["dy"], s["p"], workspace=s["ws_dw"])
    dx = api.conv2d(api.INPUT_BACKPROP, s["dy"], s["w"], s["p"])
    return {"y": y, "dw": dw, "dx": dx}


def _work_conv(case, passes=3):
    p = _conv_params(case)
    nx, nw, ny = _conv_sizes(p)
    es = 4 if case["dtype"] == "f32" else 2
    return {"bytes": passes * es * (nx + nw + ny),
            "flops": passes * 2 * ny * p.window_rows * p.window_cols * (p.channels // p.groups)}


def _run_grouped(s):
    return api.conv2d(api.FORWARD, s["x"], s["w"], s["p"], bias=s["b"], activation=api.ACT_RELU)


# ---- convolution + batch normalisation + ReLU -------------------------------------------------------


def _prepare_norm(case, seed):
    s = _prepare_conv(dict(case, stride=1), seed)
    dt, g, k = DTYPES[case["dtype"]], torch.Generator(device="cuda").manual_seed(seed + 1000003), case["features"]
    s["bn"] = api.batchnorm_params(case["batch"], case["rows"], case["cols"], k, True)
    s["beta"], s["gamma"] = _randn(g, k, dt, 0.1), (1.0 + 0.1 * torch.randn(k, device="cuda", generator=g)).to(dt)
    s["mean"], s["var"] = _randn(g, k, dt, 0.1), (2.0 + 0.2 * torch.rand(k, device="cuda", generator=g)).to(dt)
    return s


def _run_norm(s):
    p = s["p"]
    c = api.conv2d(api.FORWARD, s["x"], s["w"], p, workspace=s["ws"])
    n, mean, var = api.batchnorm_forward(c, s["beta"], s["gamma"], s["mean"], s["var"], s["bn"])
    y = api.pointwise(api.ACT_RELU, n)
    dn = api.pointwise_grad(api.ACT_RELU, y, s["dy"])
    dc, dbeta, dgamma = api.batchnorm_gradient(c, dn, s["gamma"], s["bn"])
    dw = api.conv2d(api.FILTER_BACKPROP, s["x"], dc, p, workspace=s["ws_dw"])
    dx = api.conv2d(api.INPUT_BACKPROP, dc, s["w"], p)
    return {"y": y, "mean": mean, "var": var, "dbeta": dbeta, "dgamma": dgamma, "dw": dw, "dx": dx}


def _work_norm(case):
    w = _work_conv(dict(case, stride=1))
    ny = _conv_out(_conv_params(dict(case, stride=1)))
    # normalisation 2, ReLU 2, its gradient 3, gradient of the normalisation 3 tensors of the output's size
    return {"bytes": w["bytes"] + 2 * 10 * ny, "flops": w["flops"] + 20 * ny}


# ---- classifier head ----------------------------------------------------------------------------------


def _prepare_head(case, seed):
    dt, g = DTYPES[case["dtype"]], torch.Generator(device="cuda").manual_seed(seed)
    n, hw, c, k = case["batch"], case["size"], case["channels"], case["classes"]
    dy = torch.zeros(n, k, device="cuda")
    hit = torch.randint(0, k, (n,), device="cuda", generator=g)
    dy.scatter_(1, hit[:, None], -1.0)  # the loss pulls at one class of each image, as a cross entropy does
    dy = dy + 0.05 * torch.randn(n, k, device="cuda", generator=g)
    return {"case": case, "pool": api.pool_params(n, hw, hw, c, hw, 1, False),
            "x": torch.randn(n * hw * hw * c, device="cuda", generator=g).relu().to(dt),
            "w": _randn(g, c * k, dt, (1.0 / c) ** 0.5), "b": _randn(g, k, dt, 0.1),
            "dy": (1024.0 * dy).reshape(-1).to(dt)}  # (a loss scale, as 16-bit training uses one)


def _run_head(s):
    n, c, k = s["case"]["batch"], s["case"]["channels"], s["case"]["classes"]
    f = api.pooling(api.POOL_AVERAGE, 0, s["x"], s["pool"])
    z = api.bias_add(api.matmul(f, s["w"], 1, n, c, k), s["b"], k)
    y = api.softmax(z, n, 1, 1, k)
    dz = api.softmax(y, n, 1, 1, k, gradient=s["dy"])
    dw = api.matmul(f, dz, 1, c, n, k, transpose_lhs=True)
    df = api.matmul(dz, s["w"], 1, n, k, c, transpose_rhs=True)
    dx = api.pooling(api.POOL_AVERAGE, 1, df, s["pool"])
    return {"logits": z, "y": y, "dw": dw, "dx": dx}


def _work_head(case):
    es = 4 if case["dtype"] == "f32" else 2
    n, c, k, px = case["batch"], case["channels"], case["classes"], case["size"] ** 2
    return {"bytes": es * (2 * n * c * (px + 1) + 3 * (n * c + c * k + n * k) + 2 * n * k + 5 * n * k), "flops": 6 * n * c * k}


# ---- pooling ---------------------------------------------------------------------------------------------


def _pools(case):
    args = (case["batch"], case["rows"], case["cols"], case["channels"])
    return [api.pool_params(*args, 3, 2, True), api.pool_params(*args, 2, 2, False)]


def _prepare_pool(case, seed):
    dt, g = DTYPES[case["dtype"]], torch.Generator(device="cuda").manual_seed(seed)
    pools = _pools(case)
    p = pools[0]
    x = torch.randn(p.batch * p.in_rows * p.in_cols * p.channels, device="cuda", generator=g).relu().to(dt)
    return {"pools": pools, "x": x, "dy": [_randn(g, q.batch * q.out_rows * q.out_cols * q.channels, dt) for q in pools]}


def _run_pool(s):
    out = {}
    for p, dy in zip(s["pools"], s["dy"]):
        y = api.pooling(api.POOL_MAX, 0, s["x"], p)
        out["y%d" % p.window_rows] = y
        out["dx%d" % p.window_rows] = api.pooling_max_grad(api.POOL_MAX, s["x"], y, dy, p)
    return out


def _work_pool(case):
    es = 4 if case["dtype"] == "f32" else 2
    moved = flops = 0
    for p in _pools(case):
        x, y = p.batch * p.in_rows * p.in_cols * p.channels, p.batch * p.out_rows * p.out_cols * p.channels
        moved += es * (x + y + 2 * x + 2 * y)
        flops += 2 * p.window_rows * p.window_cols * y
    return {"bytes": moved, "flops": flops}


# ---- what is measured -------------------------------------------------------------------------------------

_KINDS = {
    "net": (_prepare_net, _run_net, _work_net),
    "mobilenet": (_prepare_mobilenet, _run_mobilenet, _work_mobilenet),
    "depthwise": (_prepare_depthwise, _run_depthwise, _work_depthwise),
    "conv": (_prepare_conv, _run_conv, _work_conv),
    "norm": (_prepare_norm, _run_norm, _work_norm),
    "grouped": (_prepare_conv, _run_grouped, lambda case: _work_conv(case, 1)),
    "head": (_prepare_head, _run_head, _work_head),
    "pool": (_prepare_pool, _run_pool, _work_pool),
}


def prepare(case, seed):
    state = _KINDS[case["kind"]][0](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    return _KINDS[state["kind"]][1](state)


def work(case):
    return _KINDS[case["kind"]][2](case)


# Largest relative errors (2-norm) per kind and type: about four times what was measured against the same
# computation in float64, or, for the networks, against the library with a ten-thousandth of its inputs and
# weights moved by one unit in the last place (which is what another order of the sums does).
_TOLERANCES = {
    # measured: resnet50 5.7e-4 / 6.1e-3, vgg16 9.8e-4 in f16 and 2.1e-4 in f32
    "forward": {"f16": 4e-3, "bf16": 2.4e-2, "f32": 8e-4},
    # measured: 2.1e-3 / 1.7e-2 in the first layer's gradient, behind all the others
    "backward": {"f16": 8e-3, "bf16": 3e-2},
    # measured 1.3e-2: ReLU masks on values near zero, then a few gradients with and without them
    "train": {"f32": 3e-2},
    "mobilenet": {"f16": 8e-3},                             # measured 2.0e-3
    "depthwise": {"f16": 2e-3, "bf16": 7e-3},               # measured 4.7e-4 / 1.7e-3
    "conv": {"f16": 1.2e-3, "bf16": 9e-3, "f32": 3e-4},     # measured 2.9e-4 / 2.3e-3 / 7.7e-5 (3xTF32, 12500 terms)
    "grouped": {"f16": 1.2e-3, "bf16": 9e-3},               # measured 2.9e-4 / 2.3e-3
    "norm": {"f16": 1.6e-2, "bf16": 3e-2},                  # measured 4.4e-3 / 1.3e-2, ReLU masks again
    "head": {"f16": 2.4e-3, "bf16": 2e-2, "f32": 6e-5},     # measured 6.2e-4 / 5.1e-3 / 1.5e-5
    "pool": {"f16": 1e-4, "bf16": 4e-4, "f32": 1e-6},       # maxima are exact; sums of up to four gradients
}


def tolerance(case):
    return {"rel": _TOLERANCES[case["mode"] if case["kind"] == "net" else case["kind"]][case["dtype"]]}
