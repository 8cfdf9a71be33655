"""The work this framework is used for, as cases that can be measured.

Seven kinds of call, each through the entry points a program uses:

  scatter    perfect-spatial-hash bucketing of a batch of scans and the index of the bucket order (the data preparation
             step on its own; integer results, the same on every run)
  layer      one bucketed-attention layer in fp16 on the operator module, outputs allocated by the caller: QKV projection,
             attention, output projection
  attention  BucketSwinAttentionModule in bf16, forward or forward and backward with parameter gradients
  forward    inference of the five-stage backbone, issued kernel by kernel: from coordinates on the device, or from scan
             records in pinned host memory as a data loader delivers them; with or without per-point input features and
             the input order of the points restored
  graph      the same inference replayed as one CUDA graph, what a server does for batches of one signature
  train      forward, loss, backward and gradient buckets of the backbone (one micro-batch of a training step)
  stress     bucketing, three rounds of pooling and the matching unpools of fp32 features on heavy-tailed scenes

Scenes are LiDAR-like scans, the ground-and-blobs scan of the small configuration, or heavy-tailed voxel occupancy, made
on the device from the seed with the distributions of flash3dtransformer_b200.synthetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from flash3dtransformer_b200 import configs, graph, parallel
from flash3dtransformer_b200.layers import pooling, unpool
from flash3dtransformer_b200.layers.buck_swin import BucketSwinAttentionModule
from flash3dtransformer_b200.lib import pshattn
from flash3dtransformer_b200.psh import batching, bucket_scope, psh_main, scan_io

CHANNELS = (32, 64, 128, 256, 512)
DEPTHS = (2, 2, 2, 6, 2)
BUCKET, SCOPE = 512, 8
WINDOW = BUCKET * SCOPE


def _case(name, kind, sizes, **more):
    c = {"name": name, "kind": kind, "sizes": ",".join(str(s) for s in sizes)}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call in use: bucketing one 20,000-point scan for a per-bucket attention layer
        _case("scatter_1x20k", "scatter", [20000], scene="blobs", bucket=256, hash_op=2),
        # the CPU-runnable configuration: dim 128 = 4 heads x 32, bucket 256, fp16, 20,224 rows
        _case("layer_fp16_20k", "layer", [20224], channels=128, heads=4, bucket=256, scope=1),
        # attention layer configuration: 8 scans of 120,000 points, dim 256 = 8 heads x 32, one bucket per scope
        _case("attention_8x120k", "attention", [960000 // 512 * 512], channels=256, heads=8, bucket=512, scope=1, backward=True),
        # wider heads over the backbone's window
        _case("attention_head64", "attention", [98304], channels=512, heads=8, bucket=512, scope=8, backward=True),
        # one small scan: a robot's or a car's next frame, where the latency of the call is what counts
        _case("forward_1x20k", "forward", [20000], hash_op=2, records=False, features=False),
        # the same frame on a recorded graph
        _case("graph_1x20k", "graph", [20000], hash_op=2),
        # one full scan as the loader delivers it: fp32 records in pinned host memory
        _case("forward_1x120k_records", "forward", [119387], hash_op=2, records=True, features=False),
        # ragged scans with input features and the point order restored (per-point prediction)
        _case("forward_4_ragged_features", "forward", [120000, 47113, 131071, 88889], hash_op=2, records=False, features=True),
        # the headline batch
        _case("forward_16x120k", "forward", [120000] * 16, hash_op=2, records=False, features=False),
        # a small training micro-batch of two ragged scans
        _case("train_2_ragged", "train", [120000, 61234], hash_op=2),
        # the training configuration's micro-batch: eight scans of 200,000 points
        _case("train_8x200k", "train", [200000] * 8, hash_op=2),
        # pooling pyramid over heavy-tailed scenes of a million points, fp32 features
        _case("stress_8x1000k", "stress", [1000000] * 8, channels=128, bucket=2048, hash_op=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scans(rng, most_points, most_scenes, lo=12000, hi=140000, least_scenes=1):
    """A ragged batch: the number of scans and their mean size spread over their ranges, every scan of a size of its own."""
    n = _log(rng, least_scenes, most_scenes)
    mean = min(_log(rng, lo, hi), most_points // n)
    return [max(lo // 2, int(mean * rng.uniform(0.7, 1.0))) for _ in range(n)]


def draw(rng):
    kind = rng.choice(["scatter", "layer", "attention", "forward", "forward", "graph", "train", "stress"])
    if kind == "scatter":
        scene = rng.choice(["lidar", "lidar", "blobs", "zipf"])
        return _draw(kind, _scans(rng, 3000000, 16, 12000, 400000), scene=scene, bucket=rng.choice([256, 512, 1024]),
                     hash_op=rng.choice([1, 2, 3, 4]))
    if kind == "layer":
        bucket = rng.choice([128, 256, 512])
        scope = rng.choice([1, 2, 4])
        rows = max(1, _log(rng, 8192, 400000) // (bucket * scope)) * bucket * scope
        hd = rng.choice([16, 32, 32, 64])
        return _draw(kind, [rows], channels=hd * rng.choice([2, 4, 8]), heads=0, bucket=bucket, scope=scope, head_dim=hd)
    if kind == "attention":
        bucket = rng.choice([256, 512, 1024])
        scope = rng.choice([1, 2, 4, 8])
        hd = rng.choice([16, 32, 32, 64, 128])
        channels = hd * rng.choice([h for h in (1, 2, 4, 8, 16) if 64 <= hd * h <= 512])
        backward = rng.random() < 0.6
        most = 4e8 / (channels * max(1.0, bucket * scope / 1024.0))            # within the cost of the largest listed case
        rows = max(1, int(min(most, _log(rng, 16384, 960000))) // (bucket * scope)) * bucket * scope
        return _draw(kind, [rows], channels=channels, heads=0, bucket=bucket, scope=scope, head_dim=hd, backward=backward)
    if kind == "forward":
        return _draw(kind, _scans(rng, 1900000, 16), hash_op=rng.choice([1, 2, 2]), records=rng.random() < 0.3,
                     features=rng.random() < 0.3)
    if kind == "graph":
        return _draw(kind, _scans(rng, 250000, 4), hash_op=2)
    if kind == "train":
        return _draw(kind, _scans(rng, 1600000, 8, 60000, 200000, 2), hash_op=2)
    return _draw("stress", _scans(rng, 7900000, 8, 100000, 1000000), channels=rng.choice([32, 64, 96, 128]),
                 bucket=rng.choice([1024, 2048]), hash_op=rng.choice([1, 2]))


def _draw(kind, sizes, **more):
    c = _case("", kind, sizes, **more)
    del c["name"]
    if "head_dim" in c:
        c["heads"] = c["channels"] // c.pop("head_dim")
    return c


# ------------------------------------------------------------------------------------------------------------ inputs
def _sizes(case):
    return [int(s) for s in case["sizes"].split(",")]


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _lidar(n, g, dev):
    """64 elevation rings, uniform azimuth, range density ~ 1/r on [2, 80] m; points ring by ring along the azimuth."""
    ring = torch.randint(0, 64, (n,), generator=g, device=dev)
    az = torch.rand(n, generator=g, device=dev) * (2.0 * math.pi)
    r = 2.0 * torch.pow(40.0, torch.rand(n, generator=g, device=dev))
    order = torch.argsort(ring.double() * 8.0 + az.double())
    ring, az, r = ring[order], az[order], r[order]
    e = torch.deg2rad(torch.linspace(-25.0, 3.0, 64, device=dev))[ring]
    return torch.stack([r * torch.cos(e) * torch.cos(az), r * torch.cos(e) * torch.sin(az), r * torch.sin(e)], dim=1)


def _blobs(n, g, dev):
    """70 % ground slab, 30 % on 20 Gaussian blobs, in random order."""
    u = lambda lo, hi, *shape: torch.rand(*shape, generator=g, device=dev) * (hi - lo) + lo
    ground = int(round(0.7 * n))
    a = torch.stack([u(-25, 25, ground), u(-25, 25, ground), u(-2.0, -1.8, ground)], dim=1)
    centres = torch.stack([u(-25, 25, 20), u(-25, 25, 20), u(-2, 2, 20)], dim=1)
    b = centres[torch.arange(n - ground, device=dev) % 20] + 0.5 * torch.randn(n - ground, 3, generator=g, device=dev)
    return torch.cat([a, b])[torch.randperm(n, generator=g, device=dev)]


def _zipf(n, g, dev, seed):
    """Heavy-tailed occupancy: points per occupied 0.05 m voxel ~ Zipf(1.5) in a 100 x 100 x 8 m box."""
    rng = np.random.default_rng(seed)
    parts, total = [], 0
    while total < n:
        c = np.minimum(rng.zipf(1.5, size=max(1024, n // 8)), n)
        parts.append(c)
        total += int(c.sum())
    counts = np.concatenate(parts)
    ends = np.minimum(np.cumsum(counts), n)
    counts = np.diff(ends, prepend=0)
    counts = torch.from_numpy(counts[counts > 0]).to(dev)
    vox = torch.rand(counts.shape[0], 3, generator=g, device=dev) * torch.tensor([2000.0, 2000.0, 160.0], device=dev)
    owner = torch.repeat_interleave(torch.arange(counts.shape[0], device=dev), counts, output_size=n)
    pts = (vox.floor()[owner] + torch.rand(n, 3, generator=g, device=dev)) * 0.05
    return pts - torch.tensor([50.0, 50.0, 4.0], device=dev)


def _points(case, seed, g, dev):
    scene = case.get("scene", "zipf" if case["kind"] == "stress" else "lidar")
    out = []
    for i, n in enumerate(_sizes(case)):
        out.append(_zipf(n, g, dev, seed + 1000 * i) if scene == "zipf" else _blobs(n, g, dev) if scene == "blobs" else _lidar(n, g, dev))
    return torch.cat(out)


def _seps(case, dev):
    """The separators as a loader hands them over: on the device, with their host copy."""
    host = torch.cumsum(torch.tensor(_sizes(case), dtype=torch.int64), dim=0)
    return batching.attach_host_seps(host.to(torch.uint32).to(dev), host)


def _backbone(case, seed, dev):
    torch.manual_seed(seed)
    with torch.device(dev):
        return configs.flash3d_backbone(CHANNELS, DEPTHS, BUCKET, SCOPE, case["hash_op"],
                                        scatter_input_feat=bool(case.get("features")),
                                        restore_input_order=bool(case.get("features")))


def _scopes(rows, bucket, scope, dev):
    return torch.arange(rows // bucket, dtype=torch.int64).reshape(-1, scope).to(torch.uint32).to(dev)


def prepare(case, seed):
    dev = _device()
    g = torch.Generator(dev).manual_seed(int(seed))
    kind = case["kind"]
    s = {"case": case, "kind": kind, "dev": dev}
    if kind in ("layer", "attention"):
        rows, c, h = _sizes(case)[0], case["channels"], case["heads"]
        s["scopes"] = _scopes(rows, case["bucket"], case["scope"], dev)
        if kind == "layer":
            half = torch.float16
            s["x"] = torch.randn(rows, c, generator=g, device=dev).to(half)
            bound = 1.0 / math.sqrt(c)                                         # the default initialisation of nn.Linear
            s["w"] = [((torch.rand(o, c, generator=g, device=dev) * 2 - 1) * bound).to(half) for o in (3 * c, c)]
            s["b"] = [(torch.rand(o, generator=g, device=dev) * 2 - 1) * bound for o in (3 * c, c)]
            s["qkv"] = torch.empty(3, rows, c, dtype=half, device=dev)
            s["o"] = torch.empty(1, rows, h, c // h, dtype=half, device=dev)
            s["lse"] = torch.empty(1, rows, h, dtype=torch.float32, device=dev)
            s["out"] = torch.empty(rows, c, dtype=half, device=dev)
            return s
        torch.manual_seed(int(seed))
        with torch.device(dev):
            s["module"] = BucketSwinAttentionModule(c, h, case["bucket"])
        s["x"] = torch.randn(1, rows, c, generator=g, device=dev).to(torch.bfloat16)
        if case["backward"]:
            s["x"].requires_grad_(True)
            s["grad"] = torch.randn(1, rows, c, generator=g, device=dev).to(torch.bfloat16)
        return s
    pts = _points(case, int(seed), g, dev)
    s["coords"] = pts.to(torch.float16).contiguous()
    s["seps"] = _seps(case, dev)
    if kind == "stress":
        s["feat"] = torch.randn(pts.shape[0], case["channels"], generator=g, device=dev)
    elif kind in ("forward", "graph"):
        s["model"] = _backbone(case, int(seed), dev).eval()
        if case.get("features"):
            s["feat"] = torch.randn(pts.shape[0], CHANNELS[0], generator=g, device=dev)
        if case.get("records"):
            extra = torch.rand(pts.shape[0], 1, generator=g, device=dev)
            s["records"] = torch.cat([pts, extra], dim=1).cpu().pin_memory()
        if kind == "graph":
            s["graph"] = graph.GraphedForward(s["model"], s["coords"], s["seps"])
    elif kind == "train":
        s["model"] = _backbone(case, int(seed), dev).train()
        s["reducer"] = parallel.GradientBucketReducer(s["model"].parameters())
    return s


# ------------------------------------------------------------------------------------------------------------- calls
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _bits(t):
    return t.view(torch.int16 if t.dtype == torch.uint16 else torch.int32)


def _scatter(case, coords, seps, bucket):
    pad_to = -(-coords.shape[0] // bucket) * bucket
    scattered, buf = psh_main.batch_bucket_scatter(coords, seps, bucket, pad_to, case["hash_op"])
    return pad_to, scattered, buf


def _run_scatter(s):
    pad_to, scattered, buf = _scatter(s["case"], s["coords"], s["seps"], s["case"]["bucket"])
    out2in, in2out = psh_main.scatter_index(buf, s["seps"], pad_to)
    return {"coord": scattered.view(torch.int16), "id": _bits(buf.bucket_id), "count": _bits(buf.bucket_cntr),
            "offset": _bits(buf.bucket_offs), "cumsum": _bits(buf.bucket_cumsum), "out2in": _bits(out2in), "in2out": _bits(in2out)}


def _run_layer(s):
    rows, c = s["x"].shape
    h = s["o"].shape[2]
    pshattn.linear_bf16(s["x"], s["w"][0], s["b"][0], s["qkv"], nsplit=3)
    q, k, v = (s["qkv"][i].view(1, rows, h, c // h) for i in range(3))
    pshattn.buck_swin_fwd(q, k, v, s["o"], s["lse"], s["scopes"], s["case"]["bucket"])
    pshattn.linear_bf16(s["o"].view(rows, c), s["w"][1], s["b"][1], s["out"])
    return {"out": s["out"], "lse": s["lse"]}


def _run_attention(s):
    m = s["module"]
    if not s["case"]["backward"]:
        with torch.no_grad():
            return {"out": m(s["x"], s["scopes"])}
    params = [m.qkv.weight, m.qkv.bias, m.proj.weight, m.proj.bias]
    out = m(s["x"], s["scopes"])
    grads = torch.autograd.grad(out, [s["x"]] + params, s["grad"])
    return {"out": out.detach(), "grads": list(grads)}


def _run_forward(s):
    with torch.no_grad():
        coords, seps = s["coords"], s["seps"]
        if s["case"]["records"]:
            coords, _, seps = scan_io.collate_scans(s["records"], _sizes(s["case"]), s["dev"])
        return {"out": s["model"](coords, s.get("feat"), seps)}


def _run_graph(s):
    return {"out": s["graph"](s["coords"])}


def _run_train(s):
    red = s["reducer"]
    red.zero()
    out = s["model"](s["coords"], None, s["seps"])
    loss = out.float().square().mean()
    with red.reducing():
        loss.backward()
    red.finish()
    return {"loss": loss.detach(), "out": out.detach(), "grads": [flat for flat, _ in red.buckets]}


def _run_stress(s):
    case = s["case"]
    _, scattered, buf = _scatter(case, s["coords"], s["seps"], case["bucket"])
    feat, coords, seps, levels = s["feat"], s["coords"], s["seps"], []
    with torch.no_grad():
        for _ in range(3):                                       # sums of two rows
            red, sb = pooling.SubbuckReduceFunction.apply(coords, feat, seps, 2, 1)
            levels.append((feat, sb))
            feat, coords, seps = red, sb.reduced_coord, sb.reduced_sep
        for res, sb in reversed(levels):
            feat = unpool.AdditiveUnpoolFunction.apply(res, feat, sb, 2)
    return {"coord": scattered, "id": _bits(buf.bucket_id), "offset": _bits(buf.bucket_offs), "pooled": levels[2][0],
            "index": [_bits(sb.unpool_ind) for _, sb in levels], "out": feat}


# -------------------------------------------------------------------------------------------------------------- work
def _pooled(sizes):
    return [(n // 1024) * 512 + (n % 1024 + 1) // 2 for n in sizes]


def _levels(case):
    """Rows of the five levels of the backbone, padded as its layers pad them."""
    sizes = _sizes(case)
    rows = [-(-sum(sizes) // (6 * WINDOW)) * 6 * WINDOW]
    for _ in CHANNELS[1:]:
        sizes = _pooled(sizes)
        rows.append(-(-sum(sizes) // WINDOW) * WINDOW)
    return rows


def _backbone_work(case):
    """(projection flops, attention flops, parameters) of one forward."""
    proj = attn = params = 0.0
    rows = _levels(case)
    for i, (n, c, d) in enumerate(zip(rows, CHANNELS, DEPTHS)):
        blocks = 2 * d
        proj += blocks * 2.0 * n * 16 * c * c
        attn += blocks * 4.0 * n * WINDOW * c
        params += blocks * (16.0 * c * c + 17 * c)
        if i + 1 < len(rows):
            up = CHANNELS[i + 1]
            proj += 2.0 * n * c * up * 2 + 2.0 * rows[i + 1] * up * c              # pooling, skip and unpooling projections
            params += 3.0 * c * up
    proj += 2.0 * rows[-1] * CHANNELS[-1] ** 2
    params += CHANNELS[-1] ** 2
    return proj, attn, params


def work(case):
    sizes = _sizes(case)
    n, kind = float(sum(sizes)), case["kind"]
    if kind == "scatter":
        return {"bytes": 26.0 * n, "flops": 0.0}                 # 6 read; 2 id, 4 offset, 6 rows, 8 indices written
    if kind in ("layer", "attention"):
        c, h = case["channels"], case["heads"]
        window = case["bucket"] * case["scope"]
        proj, attn = 8.0 * n * c * c, 4.0 * n * window * c
        if case.get("backward"):
            return {"bytes": 8.0 * n * c + 4 * 4.0 * c * c + 4 * 4.0 * c * c, "flops": 3 * proj + 3.5 * attn}
        return {"bytes": 4.0 * n * c + (4.0 * n * h if kind == "layer" else 0.0) + 2 * 4.0 * c * c, "flops": proj + attn}
    if kind in ("forward", "graph", "train"):
        proj, attn, params = _backbone_work(case)
        out_rows = n if case.get("features") else float(_levels(case)[0])
        nbytes = 6.0 * n + 2.0 * out_rows * CHANNELS[0] + 4.0 * params
        if case.get("features"):
            nbytes += 4.0 * n * CHANNELS[0]
        if case.get("records"):
            nbytes += 10.0 * n
        if kind == "train":
            return {"bytes": nbytes + 4.0 * params, "flops": 3 * proj + 3.5 * attn}
        return {"bytes": nbytes, "flops": proj + attn}
    c, total, rows = case["channels"], 18.0 * n, sizes
    for _ in range(3):
        nxt = _pooled(rows)
        up, down = float(sum(rows)), float(sum(nxt))
        total += 4.0 * c * (up + down) + 6.0 * (up + down) + 8.0 * down               # pooling: features, coordinates, index
        total += 4.0 * c * (2 * up + down) + 8.0 * down                               # unpooling
        rows = nxt
    return {"bytes": total, "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind == "scatter":
        return "exact"
    if kind == "stress":
        return {"rel": 1e-6, "max": 1e-5}                        # fp32 sums of two values, then one addition a level
    if kind == "layer":
        return {"rel": 1e-3, "max": 2e-2}                        # fp16: three rounded stages
    if kind == "attention":
        return {"rel": 1e-2, "max": 1e-1}                        # bf16: three rounded stages, gradients through them
    if kind == "train":
        # bf16 gradients through 28 blocks, forward and back; the gradients of the pooling norms are sums that nearly cancel,
        # so single entries move by a good part of a bucket's root mean square from one order of addition to another
        return {"rel": 2e-2, "max": 0.95}
    return {"rel": 1e-2, "max": 1.5e-1}                          # bf16: 28 blocks, five levels
