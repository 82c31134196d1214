"""Timed cases of the operator path: what a point-cloud model has these operators do, at real sizes.

Every case is one pass through the public entry points (``torkit3d_b200.ops`` and ``torkit3d_b200.layers``) as a
training step or a preprocessing step calls them; where the path has a backward pass the pass includes it and the
gradients are among the outputs.  All tensors are float32, the type such models train in (float64 is served by the
operators for gradient checks).  Coordinates come in both layouts ([B,N,3]: ``transpose`` false, [B,3,N]: true) and
indices in both widths where the entry point offers it.

``op`` is one of

chamfer  chamfer_distance and its gradients for both clouds under per-point upstream gradients
knn      knn_points
fps      sample_farthest_points
group    ball_query + group_points and the feature gradient, operator by operator
sa       the set-abstraction front end: sample_and_gather + set_abstraction_group and the feature and coordinate gradients
interp   knn_points(k=3) + three_nn_weight + interpolate_feature and the feature gradient, operator by operator
fp       three_nn_interpolate (the fused feature propagation) and the feature gradient
edge     knn on the features + get_edge_feature and the feature gradient (a dynamic-graph EdgeConv layer)
"""
import math

import torch

from torkit3d_b200 import layers, ops


def listed():
    return [
        # a reconstruction loss on object-sized clouds: the smallest call, bound by latency and launches
        dict(name="chamfer_1k", op="chamfer", B=2, N=1024, M=1024, points="uniform", transpose=False),
        # a completion loss: a ragged prediction against a larger ragged target, channel-first tensors
        dict(name="chamfer_ragged", op="chamfer", B=24, N=2500, M=4099, points="mixture", transpose=True),
        # the benchmark's training step: loss gradients on a batch of dense clouds
        dict(name="chamfer_16k", op="chamfer", B=64, N=16384, M=16384, points="mixture", transpose=False),
        # neighbourhoods of 16 points, queries and keys of the same size (the KNN configuration of the benchmark)
        dict(name="knn_16", op="knn", B=16, N=4096, M=4096, K=16, points="normal", transpose=False, same=False,
             index32=False),
        # neighbourhoods of 32 points of a subsampled cloud in the full one (a size of the operator benchmarks)
        dict(name="knn_32", op="knn", B=32, N=2048, M=8192, K=32, points="sphere", transpose=True, same=False,
             index32=True),
        # the first sampling stage of a classification model on dense objects
        dict(name="fps_8k", op="fps", B=32, N=8192, S=1024, points="sphere", transpose=False),
        # subsampling whole scenes: few large clouds, many samples
        dict(name="fps_scene", op="fps", B=4, N=65536, S=2048, points="box", transpose=True),
        # ball query + grouping of a first set-abstraction stage, forward and backward, operator by operator
        dict(name="group_8k", op="group", B=32, N=8192, M=1024, C=64, K=32, hits=20.5, points="sphere"),
        # a second set-abstraction stage through the fused front end: small clouds, wide features, dense balls
        dict(name="sa_512", op="sa", B=32, N=512, M=128, C=128, K=64, hits=20.0, points="sphere"),
        # an ordinary feature propagation stage, operator by operator
        dict(name="interp_4k", op="interp", B=16, N=4096, M=1024, C=256, points="sphere"),
        # feature propagation to every point of large scenes, the largest call
        dict(name="fp_scene", op="fp", B=8, N=131072, M=32768, C=128, points="box"),
        # a dynamic-graph EdgeConv layer: neighbours in feature space, edge features, their gradients
        dict(name="edge_1k", op="edge", B=32, N=1024, C=64, K=20),
    ]


_POINTS = ("uniform", "normal", "mixture", "sphere", "box")


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _fit(rng, high, per_unit, limit):
    """A batch size of 1 to ``high`` whose work (``per_unit`` each) stays below ``limit``."""
    return _log_int(rng, 1, max(1, min(high, int(limit // per_unit))))


def draw(rng):
    op = rng.choice(("chamfer", "chamfer", "knn", "knn", "fps", "fps", "group", "sa", "interp", "fp", "edge"))
    points, flip = rng.choice(_POINTS), rng.random() < 0.5
    if op == "chamfer":
        N, M = _log_int(rng, 512, 16384), _log_int(rng, 512, 16384)
        return dict(op=op, B=_fit(rng, 64, N * M, 1.2e10), N=N, M=M, points=points, transpose=flip)
    if op == "knn":
        N, M = _log_int(rng, 512, 16384), _log_int(rng, 512, 16384)
        return dict(op=op, B=_fit(rng, 32, N * M, 2e9), N=N, M=N if flip else M, K=_log_int(rng, 3, 64), points=points,
                    transpose=rng.random() < 0.5, same=flip, index32=rng.random() < 0.3)
    if op == "fps":
        N = _log_int(rng, 512, 65536)
        return dict(op=op, B=_fit(rng, 64, N, 262144), N=N, S=_log_int(rng, 64, min(2048, N // 4)), points=points,
                    transpose=flip)
    if op in ("group", "sa"):
        N = _log_int(rng, 512, 16384)
        M, C, K = max(32, int(N * rng.uniform(0.1, 0.5))), _log_int(rng, 16, 256), _log_int(rng, 8, 64)
        return dict(op=op, B=_fit(rng, 32, M * C * K + C * N, 8e7), N=N, M=M, C=C, K=K,
                    hits=round(K * rng.uniform(0.4, 1.5), 1), points=rng.choice(("sphere", "uniform", "box")))
    if op in ("interp", "fp"):
        N, ratio, C = _log_int(rng, 1024, 131072), rng.uniform(0.15, 0.5), _log_int(rng, 16, 256)
        return dict(op=op, B=_fit(rng, 16, N * max(C, 32) * (1 + N / 16384), 1.2e8), N=N, M=int(N * ratio), C=C,
                    points=points)
    N, C = _log_int(rng, 256, 2048), _log_int(rng, 16, 128)
    return dict(op=op, B=_fit(rng, 32, N * C * max(40, N // 16), 2e8), N=N, C=C, K=_log_int(rng, 8, 40))


def _cloud(kind, B, N, g, centres=None):
    """[B,N,3] points as the benchmark's configurations draw them, scattered in memory as sampled clouds are."""
    dev = g.device
    if kind == "uniform":
        return torch.rand(B, N, 3, generator=g, device=dev) * 2 - 1
    if kind == "normal":
        return torch.randn(B, N, 3, generator=g, device=dev)
    if kind == "box":  # a room: 10 x 10 x 3 m
        return torch.rand(B, N, 3, generator=g, device=dev) * torch.tensor([10.0, 10.0, 3.0], device=dev)
    if kind == "mixture":  # 8 blobs per cloud, shared by the two clouds of a pair
        pick = torch.randint(0, 8, (B, N, 1), generator=g, device=dev).expand(-1, -1, 3)
        return torch.gather(centres, 1, pick) + 0.1 * torch.randn(B, N, 3, generator=g, device=dev)
    p = torch.randn(B, N, 3, generator=g, device=dev)  # sphere: a scanned surface with noise
    return p / p.norm(dim=2, keepdim=True) + 0.01 * torch.randn(B, N, 3, generator=g, device=dev)


def _radius(case):
    """The ball radius with the wanted mean number of hits in the region that a cloud fills."""
    share = case["hits"] / case["N"]
    if case["points"] == "sphere":
        return 2 * math.sqrt(share)  # a cap of radius r covers r^2 / 4 of the unit sphere
    volume = 8.0 if case["points"] == "uniform" else 300.0
    return (share * volume * 3 / (4 * math.pi)) ** (1 / 3)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    op, B, N = case["op"], case["B"], case["N"]
    s = dict(case=case)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    if op == "edge":
        s.update(x=randn(B, case["C"], N).requires_grad_(), grad=randn(B, 2 * case["C"], N, case["K"]))
        return s
    centres = torch.rand(B, 8, 3, generator=g, device="cuda") * 2 - 1
    a = _cloud(case["points"], B, N, g, centres)
    if op in ("chamfer", "knn"):
        b = a if case.get("same") else _cloud(case["points"], B, case["M"], g, centres)
        if case["transpose"]:
            a, b = (t.transpose(1, 2).contiguous() for t in (a, b))
        if op == "chamfer":
            a.requires_grad_(), b.requires_grad_()
            # upstream gradients of a weighted mean over the points
            s.update(grad=tuple(torch.rand(B, n, generator=g, device="cuda") / (B * n) for n in (N, case["M"])))
        s.update(a=a, b=b)
        return s
    if op == "fps":
        s.update(a=a.transpose(1, 2).contiguous() if case["transpose"] else a)
        return s
    C, M = case["C"], case["M"]
    a = a.transpose(1, 2).contiguous()  # [B,3,N], as the layers pass coordinates around
    if op in ("group", "sa"):
        feature = randn(B, C, N).requires_grad_()
        s.update(a=a, feature=feature, radius=_radius(case))
        if op == "group":
            # a random subset of an i.i.d. cloud stands for its sampled centres
            s.update(centre=a[:, :, torch.randperm(N, generator=g, device="cuda")[:M]].contiguous(),
                     grad=randn(B, C, M, case["K"]))
        else:
            a.requires_grad_()
            s.update(grad=randn(B, C + 3, M, case["K"]))
        return s
    key = _cloud(case["points"], B, M, g, centres).transpose(1, 2).contiguous()
    s.update(a=a, key=key, feature=randn(B, C, M).requires_grad_(), grad=randn(B, C, N))
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "chamfer":
        d1, d2 = ops.chamfer_distance(s["a"], s["b"], transpose=case["transpose"])
        return (d1, d2) + torch.autograd.grad((d1, d2), (s["a"], s["b"]), s["grad"])
    if op == "knn":
        if case["index32"]:
            return ops.knn_points(s["a"], s["b"], case["K"], transpose=case["transpose"], index_dtype=torch.int32)
        return ops.knn_points(s["a"], s["b"], case["K"], transpose=case["transpose"])
    if op == "fps":
        return ops.sample_farthest_points(s["a"], case["S"], case["transpose"])
    if op == "group":
        index = ops.ball_query(s["centre"], s["a"], s["radius"], case["K"])
        out = ops.group_points(s["feature"], index)
        return (index, out) + torch.autograd.grad(out, s["feature"], s["grad"])
    if op == "sa":
        index, centre = layers.sample_and_gather(s["a"], case["M"])
        out = layers.set_abstraction_group(s["a"], centre, s["feature"], s["radius"], case["K"])
        return (index, centre, out) + torch.autograd.grad(out, (s["a"], s["feature"]), s["grad"])
    if op == "interp":
        distance, index = ops.knn_points(s["a"], s["key"], 3, transpose=True)
        weight = ops.three_nn_weight(distance)
        out = ops.interpolate_feature(s["feature"], index, weight)
        return (index, weight, out) + torch.autograd.grad(out, s["feature"], s["grad"])
    if op == "fp":
        out = layers.three_nn_interpolate(s["a"], s["key"], s["feature"])
        return (out,) + torch.autograd.grad(out, s["feature"], s["grad"])
    distance, index = ops.knn(s["x"].detach(), s["x"].detach(), case["K"], transpose=True)
    edge = ops.get_edge_feature(s["x"], s["x"], index)
    return (distance, index, edge) + torch.autograd.grad(edge, s["x"], s["grad"])


def work(case):
    """Inputs read once, outputs written once; one distance (8 flop) for each neighbour or sample that is returned (an
    exact search need not look at every pair), the arithmetic of the sums."""
    op, B, N, K = case["op"], case["B"], case["N"], case.get("K", 3)
    M, C = case.get("M", N), case.get("C", 0)
    if op == "chamfer":
        return {"bytes": B * (N + M) * (12 + 4 + 4 + 12), "flops": B * (N + M) * (8 + 12)}
    if op == "knn":
        return {"bytes": B * (12 * (N + (0 if case["same"] else M)) + N * K * (8 if case["index32"] else 12)),
                "flops": 8 * B * N * K}
    if op == "fps":
        return {"bytes": B * (12 * N + 8 * case["S"]), "flops": 8 * B * N}
    if op == "group":
        return {"bytes": B * (12 * (N + M) + 8 * M * K + 8 * C * N + 8 * C * M * K), "flops": B * (8 + C) * M * K}
    if op == "sa":
        return {"bytes": B * (24 * N + 20 * M + 8 * C * N + 8 * (C + 3) * M * K), "flops": B * (11 + C) * M * K}
    if op == "interp":
        return {"bytes": B * (12 * (N + M) + 36 * N + 8 * C * (N + M)), "flops": B * N * (3 * 11 + 12 * C)}
    if op == "fp":
        return {"bytes": B * (12 * (N + M) + 8 * C * (N + M)), "flops": B * N * (3 * 11 + 12 * C)}
    return {"bytes": B * N * (8 * C + 12 * K + 16 * C * K), "flops": B * N * K * (3 * C + 2 * C)}


def tolerance(case):
    """Whole values are exact.  Gradients are float32 sums in any order: against the same sums in float64 they measured
    up to rel 2e-7 and max 4.6e-6 (dense balls, up to a hundred terms each); stated are about four times that."""
    return {"rel": 1e-6, "max": 2e-5, "differ": 0.0}
