"""What a network that runs on these layer kernels has them do, as cases to be timed.

Kinds (a case names one and gives its sizes; tensors are fp32 [n][c][h][w], the one type of the library):

  infer      batch norm with running statistics (+ residual) + activation, one call
  train      batch norm with batch statistics + its activations, forward and then backward with all per-channel gradients;
             through the C ABI's binding ("calls") or through the layer objects that a scheduler holds ("objects")
  pool       max subsampling with argmax, forward and then backward: fused behind batch norm -> residual add -> ReLU
             (the tail of a residual block), or the stand-alone layer
  softmax    channel softmax, forward and then backward; with the negative log likelihood fused behind it, or the plain layer
  optimizer  the update of all weight chunks of a network

Every pass takes its buffers, workspaces and objects as a training or serving loop would: made once, in prepare().
"""
import math

import torch

EPS = 1e-5
WEIGHT_COUNT_PER_LAYER = 9   # a 3x3 convolution: width * width * 9 weights


def listed():
    return [
        # one image through the end of a residual block: launch and host latency
        {"name": "infer 1 image", "kind": "infer", "n": 1, "c": 64, "h": 32, "w": 32, "act": "relu", "residual": True},
        # an ordinary serving batch behind a convolution
        {"name": "infer batch 64", "kind": "infer", "n": 64, "c": 64, "h": 32, "w": 32, "act": "relu", "residual": False},
        # scoring a large data set in slabs of 2 GiB
        {"name": "infer 2 GiB", "kind": "infer", "n": 1024, "c": 128, "h": 64, "w": 64, "act": "tanh", "residual": False},
        # a training step of a mid-network layer at the batch of one GPU
        {"name": "train 28x28", "kind": "train", "n": 256, "c": 256, "h": 28, "w": 28, "act": "prelu_elu", "through": "calls"},
        # the same layer of a small network, driven object by object
        {"name": "train small, objects", "kind": "train", "n": 32, "c": 64, "h": 16, "w": 16, "act": "prelu_elu", "through": "objects"},
        # the last stage of an image network: planes that are not whole vectors
        {"name": "train 7x7", "kind": "train", "n": 256, "c": 512, "h": 7, "w": 7, "act": "relu", "through": "calls"},
        # odd planes and an ordinary batch
        {"name": "train 27x27", "kind": "train", "n": 128, "c": 96, "h": 27, "w": 27, "act": "relu", "through": "calls"},
        # the tail of the first residual stage, with its pooling
        {"name": "pool 56x56 fused", "kind": "pool", "n": 256, "c": 64, "h": 56, "w": 56, "win": 3, "fused": True},
        # the stand-alone subsampling layer on ragged planes
        {"name": "pool 55x55", "kind": "pool", "n": 64, "c": 96, "h": 55, "w": 55, "win": 3, "fused": False},
        # the classifier at the end of a training step
        {"name": "softmax 256 rows", "kind": "softmax", "n": 256, "c": 1000, "h": 1, "w": 1, "loss": True},
        # per-pixel classes of a segmentation network
        {"name": "softmax pixels", "kind": "softmax", "n": 32, "c": 21, "h": 128, "w": 128, "loss": False},
        # one step of the optimiser over a whole network
        {"name": "optimizer", "kind": "optimizer", "layers": 20, "width": 256, "momentum": "vanilla"},
    ]


# ---------------------------------------------------------------------------------------------------------------------
# drawn cases


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _channels(rng, lo, hi):
    c = int(round(_log(rng, lo, hi)))
    if rng.random() < 0.5:
        c = max(8, c // 8 * 8)   # what networks mostly have; the other half of the draws keeps odd counts
    return max(lo, min(hi, c))


def _plane(rng, lo, hi):
    h = max(lo, min(hi, int(round(_log(rng, lo, hi)))))
    if rng.random() < 0.7:
        return h, h
    return h, max(lo, min(hi, int(round(_log(rng, max(lo, h // 2), min(hi, 2 * h))))))


def _entries(rng, elements, c, h, w, most):
    return max(1, min(most, int(round(elements / (c * h * w)))))


def draw(rng):
    kind = rng.choice(["infer", "train", "pool", "softmax", "optimizer"])
    while True:
        case = _draw_of(rng, kind)
        if case is not None:
            return case


def _draw_of(rng, kind):
    if kind == "infer":
        e = _log(rng, 1 << 14, 1 << 28)
        c = _channels(rng, 3, 2048)
        h, w = _plane(rng, 1, 128)
        case = {"kind": kind, "n": _entries(rng, e, c, h, w, 8192), "c": c, "h": h, "w": w,
                "act": rng.choice(["relu", "relu", "relu", "prelu", "elu", "tanh", "sigmoid", "none"]), "residual": rng.random() < 0.4}
        return case if 1 << 12 <= _elements(case) <= 1 << 29 else None
    if kind == "train":
        e = _log(rng, 1 << 15, 1 << 26)
        c = _channels(rng, 3, 2048)
        h, w = _plane(rng, 1, 112)
        case = {"kind": kind, "n": _entries(rng, e, c, h, w, 1024), "c": c, "h": h, "w": w,
                "act": rng.choice(["relu", "relu", "relu", "prelu_elu", "prelu", "elu", "tanh", "none"]), "through": "calls"}
        if case["act"] in ("relu", "prelu_elu") and rng.random() < 0.3:
            case["through"] = "objects"
        # batch statistics need a batch
        return case if 1 << 13 <= _elements(case) <= 1 << 26 and case["n"] >= 4 and case["n"] * h * w >= 64 else None
    if kind == "pool":
        e = _log(rng, 1 << 15, 1 << 26)
        c = _channels(rng, 3, 1024)
        h, w = _plane(rng, 6, 112)
        case = {"kind": kind, "n": _entries(rng, e, c, h, w, 1024), "c": c, "h": h, "w": w, "win": rng.choice([3, 3, 2]), "fused": rng.random() < 0.5}
        return case if 1 << 13 <= _elements(case) <= 1 << 26 else None
    if kind == "softmax":
        e = _log(rng, 1 << 14, 1 << 26)
        if rng.random() < 0.5:
            c, h, w, most = int(round(_log(rng, 10, 32000))), 1, 1, 65536
        else:
            c, most = int(round(_log(rng, 2, 160))), 512
            h, w = _plane(rng, 8, 128)
        case = {"kind": kind, "n": _entries(rng, e, c, h, w, most), "c": c, "h": h, "w": w, "loss": rng.random() < 0.6}
        return case if 1 << 12 <= _elements(case) <= 1 << 26 else None
    case = {"kind": kind, "layers": int(round(_log(rng, 2, 64))), "width": int(round(_log(rng, 16, 512))),
            "momentum": rng.choice(["none", "vanilla", "vanilla", "nesterov", "adam"])}
    return case if _weights(case) <= 1 << 26 else None


# ---------------------------------------------------------------------------------------------------------------------
# sizes


def _elements(case):
    return case["n"] * case["c"] * case["h"] * case["w"]


def _pooled(case):
    return case["n"] * case["c"] * ((case["h"] - case["win"]) // 2 + 1) * ((case["w"] - case["win"]) // 2 + 1)


def _chunk_sizes(case):
    w = case["width"]
    return [w * w * WEIGHT_COUNT_PER_LAYER] + [w] * 5   # a convolution's weights and bias; gamma, beta, mean, inverse sigma


def _weights(case):
    return case["layers"] * sum(_chunk_sizes(case))


def work(case):
    kind = case["kind"]
    if kind == "optimizer":
        # data and gradient are read and written, and so is each buffer that the momentum type keeps
        state = {"none": 0, "vanilla": 1, "nesterov": 1, "adam": 2}[case["momentum"]]
        flops = {"none": 5, "vanilla": 7, "nesterov": 10, "adam": 18}[case["momentum"]]
        return {"bytes": _weights(case) * 4 * (4 + 2 * state), "flops": _weights(case) * flops}
    e = _elements(case)
    if kind == "infer":
        return {"bytes": e * (12 if case["residual"] else 8), "flops": e * 6}
    if kind == "train":
        return {"bytes": e * 20, "flops": e * 24}   # x -> y; x, dy -> dx
    if kind == "pool":
        p = _pooled(case)
        if case["fused"]:
            # x, residual -> z, pooled, argmax; dpooled, argmax, z -> dx, dresidual
            return {"bytes": e * 24 + p * 16, "flops": e * 20}
        return {"bytes": e * 8 + p * 16, "flops": e * 12}
    pixels = case["n"] * case["h"] * case["w"]
    if case["loss"]:
        return {"bytes": e * 24 + pixels * 4, "flops": e * 20}   # logits, targets -> p, err; p, targets -> dlogits
    return {"bytes": e * 20, "flops": e * 14}                    # x -> y; dy, y -> dx


def tolerance(case):
    kind = case["kind"]
    if kind == "pool":
        return "exact"
    if kind == "infer":
        # products and sums rounded one by one are the same everywhere; the exponentials are good to some units in the last place
        return {"rel": 1e-5} if case["act"] in ("elu", "tanh", "sigmoid") else "exact"
    if kind == "optimizer":
        return {"rel": 1e-6}
    return {"rel": 1e-5}


# ---------------------------------------------------------------------------------------------------------------------
# inputs and passes


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, shape, mean=0.0, std=1.0):
    return torch.empty(shape, device="cuda").normal_(mean, std, generator=g)


def _uniform(g, shape, lo, hi):
    return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=g)


def _bn_weights(g, c):
    """gamma, beta, running mean, running inverse sigma."""
    return (_uniform(g, c, 0.5, 1.5), _normal(g, c, 0.0, 0.1), _normal(g, c, 0.0, 0.1), (_uniform(g, c, 0.5, 2.0) + EPS).rsqrt())


def _off_the_kink(x, gamma, beta):
    """A rectifier's derivative jumps where the batch-norm output is 0, and two correct evaluations of an output of 1e-7 may be on
    different sides. The few such elements of x move off by 1e-3 of the channel's deviation."""
    dims = [0, 2, 3]
    for lo in range(0, x.shape[1], 64):
        part = x[:, lo:lo + 64]
        var, mean = torch.var_mean(part.double(), dim=dims, correction=0, keepdim=True)
        sigma = (var + EPS).sqrt()
        scale = gamma[lo:lo + 64].double().view(1, -1, 1, 1) / sigma
        u = (part - mean) * scale + beta[lo:lo + 64].double().view(1, -1, 1, 1)
        part.add_(((u.abs() < 2e-5) * (1e-3 * sigma)).float())


def _acts(capi, name, slope):
    return {"none": lambda: [], "relu": lambda: [capi.relu()], "prelu": lambda: [capi.prelu(slope)], "elu": lambda: [capi.elu()],
            "tanh": lambda: [capi.tanh()], "sigmoid": lambda: [capi.sigmoid()],
            "prelu_elu": lambda: [capi.prelu(slope), capi.elu()]}[name]()


def prepare(case, seed):
    from nnforge_b200 import capi
    g = _generator(seed)
    state = {"kind": case["kind"], "case": case, "capi": capi}
    state.update({"infer": _prepare_infer, "train": _prepare_train, "pool": _prepare_pool, "softmax": _prepare_softmax,
                  "optimizer": _prepare_optimizer}[case["kind"]](capi, case, g))
    return state


def run(state):
    return _RUN[state["kind"]](state["capi"], state)


def _shape(case):
    return case["n"], case["c"], case["h"], case["w"]


def _prepare_infer(capi, case, g):
    shape = _shape(case)
    slope = _uniform(g, case["c"], 0.0, 0.3)
    x = _normal(g, shape)
    return {"x": x, "bn": _bn_weights(g, case["c"]), "residual": _normal(g, shape) if case["residual"] else None, "slope": slope,
            "acts": _acts(capi, case["act"], slope), "y": torch.empty_like(x)}


def _run_infer(capi, s):
    capi.bn_infer_act(s["y"], s["x"], bn=s["bn"], residual=s["residual"], acts=s["acts"])
    return s["y"]


def _prepare_train(capi, case, g):
    n, c, h, w = shape = _shape(case)
    slope = _uniform(g, c, 0.0, 0.3)
    x, dy = _normal(g, shape, 0.5, 2.0), _normal(g, shape)
    weights = _bn_weights(g, c)
    if case["act"] in ("relu", "prelu", "prelu_elu"):
        _off_the_kink(x, weights[0], weights[1])
    s = {"x": x, "dy": dy, "weights": weights, "slope": slope, "y": torch.empty_like(x), "dx": torch.empty_like(x),
         "grads": [torch.zeros(c, device="cuda") for _ in range(5)], "through": case["through"]}
    if case["through"] == "calls":
        s.update(acts=_acts(capi, case["act"], slope), saved=torch.empty(2 * c, device="cuda"), sums=torch.empty(2 * c, device="cuda"),
                 bsums=torch.empty(3 * c, device="cuda"),
                 workspace=torch.empty(capi.bn_train_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda"))
        return s
    from nnforge_b200 import host
    spec = "bn BatchNorm x eps=%r\n" % EPS + {"relu": "relu ReLU bn slope=0\n", "prelu_elu": "prelu PReLU bn\nelu ELU prelu\n"}[case["act"]]
    net = host.Net(spec, {"x": (c, w, h)}, training=True)
    head = net.objects[0]
    working = max(head.get_temporary_working_fixed_buffer_size(a) for a in (host.FORWARD, host.BACKWARD_DATA_AND_WEIGHTS))
    has_slope = case["act"] != "relu"
    s.update(net=net, head=head, chunks=list(weights) + ([slope] if has_slope else []), gradients=s["grads"][:5 if has_slope else 4],
             working=torch.empty(max(working, 16), dtype=torch.uint8, device="cuda"),
             fixed=torch.empty(head.get_temporary_fixed_buffer_size() // 4, device="cuda"))
    return s


def _run_train(capi, s):
    if s["through"] == "objects":
        return _run_train_objects(s)
    gamma, beta, mean, invsigma = s["weights"]
    capi.bn_train_fwd(s["y"], s["saved"], s["sums"], s["x"], gamma, beta, EPS, s["acts"], workspace=s["workspace"])
    grads = s["grads"]
    capi.bn_train_bwd(s["dx"], s["bsums"], s["dy"], s["x"], gamma, beta, s["saved"], s["acts"], grad_gamma=grads[0], grad_beta=grads[1],
                      grad_mean=grads[2], grad_invsigma=grads[3], grad_slope=grads[4] if "prelu" in s["case"]["act"] else None, mean=mean,
                      invsigma=invsigma, entry_count=float(s["x"].shape[0]), workspace=s["workspace"])
    return s["y"], s["dx"], s["saved"], grads


def _run_train_objects(s):
    head, followers, n = s["head"], s["net"].objects[1:], s["x"].shape[0]
    head.enqueue_forward_propagation([s["y"]], s["chunks"], [s["x"]], n, temporary_working_fixed_buffer=s["working"], temporary_fixed_buffer=s["fixed"])
    for o in followers:
        o.enqueue_forward_propagation([s["y"]], [], [s["y"]], n)
    for o in reversed(followers):
        o.enqueue_backward_data_propagation(0, s["dy"], s["dy"], [], [None], None, n)
    head.enqueue_backward_data_and_weights_propagation([s["dx"]], s["dy"], s["gradients"], s["chunks"], [s["x"]], None, n,
                                                       temporary_working_fixed_buffer=s["working"], temporary_fixed_buffer=s["fixed"])
    return s["y"], s["dx"], s["fixed"], s["grads"]


def _prepare_pool(capi, case, g):
    n, c, h, w = shape = _shape(case)
    pool = capi.pool((case["win"], case["win"]), (2, 2))
    oh, ow = capi.pool_out_shape(h, w, pool)
    x = _normal(g, shape)
    s = {"pool": pool, "x": x, "pooled": torch.empty((n, c, oh, ow), device="cuda"),
         "argmax": torch.empty((n, c, oh, ow), dtype=torch.int32, device="cuda"), "dpooled": _normal(g, (n, c, oh, ow)), "dx": torch.empty_like(x)}
    if case["fused"]:
        s.update(residual=_normal(g, shape), bn=_bn_weights(g, c), z=torch.empty_like(x), dresidual=torch.empty_like(x))
    return s


def _run_pool(capi, s):
    if s["case"]["fused"]:
        capi.bn_add_relu_maxpool_fwd(s["z"], s["pooled"], s["argmax"], s["x"], s["residual"], s["bn"], 0.0, s["pool"])
        capi.bn_add_relu_maxpool_bwd(s["dx"], s["dresidual"], s["dpooled"], s["argmax"], s["z"], s["bn"][0], s["bn"][3], 0.0, s["pool"])
        return s["z"], s["pooled"], s["argmax"], s["dx"], s["dresidual"]
    capi.maxpool_fwd(s["pooled"], s["argmax"], s["x"], s["pool"])
    capi.maxpool_bwd(s["dx"], s["dpooled"], s["argmax"], s["pool"])
    return s["pooled"], s["argmax"], s["dx"]


def _prepare_softmax(capi, case, g):
    n, c, h, w = shape = _shape(case)
    x = _normal(g, shape, 0.0, 3.0 if h * w == 1 else 2.0)
    s = {"x": x, "y": torch.empty_like(x), "dx": torch.empty_like(x)}
    if case["loss"]:
        labels = torch.randint(0, c, (n, 1, h, w), device="cuda", generator=g)
        s.update(targets=torch.zeros(shape, device="cuda").scatter_(1, labels, 1.0), err=torch.empty((n, 1, h, w), device="cuda"))
    else:
        s.update(dy=_normal(g, shape))
    return s


def _run_softmax(capi, s):
    if s["case"]["loss"]:
        capi.softmax_nll_fwd(s["y"], s["err"], s["x"], s["targets"])
        capi.softmax_nll_bwd(s["dx"], s["y"], s["targets"])
        return s["y"], s["err"], s["dx"]
    capi.softmax_fwd(s["y"], s["x"])
    capi.softmax_bwd(s["dx"], s["dy"], s["y"])
    return s["y"], s["dx"]


def _prepare_optimizer(capi, case, g):
    sizes = _chunk_sizes(case) * case["layers"]
    starts, total = [], 0
    for size in sizes:
        starts.append(total)
        total += -(-size // 64) * 64   # chunks start on 256-byte boundaries, as allocations do
    kept = {"none": 0, "vanilla": 1, "nesterov": 1, "adam": 2}[case["momentum"]]
    data, gradient = _normal(g, total, 0.0, 0.05), _normal(g, total, 0.0, 0.01)
    previous = [_normal(g, total, 0.0, 1e-4).abs_() for _ in range(kept)]
    changes = torch.zeros(len(sizes), dtype=torch.float64, device="cuda")
    parts = []
    for k, (start, size) in enumerate(zip(starts, sizes)):
        part = {"data": data[start:start + size], "gradient": gradient[start:start + size], "update_accum": changes[k:k + 1],
                "learning_rate": 0.01, "weight_decay": 1e-4 if size > case["width"] else 0.0}
        for name, t in zip(("prev_upd", "prev_upd2"), previous):
            part[name] = t[start:start + size]
        parts.append(part)
    momentum = {"none": capi.MOMENTUM_NONE, "vanilla": capi.MOMENTUM_VANILLA, "nesterov": capi.MOMENTUM_NESTEROV, "adam": capi.MOMENTUM_ADAM}
    return {"data": data, "gradient": gradient, "previous": previous, "changes": changes, "parts": parts, "momentum": momentum[case["momentum"]],
            "iteration": 0}


def _run_optimizer(capi, s):
    s["iteration"] += 1
    capi.apply_gradient(s["parts"], s["momentum"], normalizer=1.0 / 256, iteration_id=s["iteration"])
    return s["data"], s["gradient"], s["previous"], s["changes"]


_RUN = {"infer": _run_infer, "train": _run_train, "pool": _run_pool, "softmax": _run_softmax, "optimizer": _run_optimizer}
