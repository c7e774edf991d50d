"""The work this router is measured on: cases over its public entry points.

Four families, each over the range of sizes it meets in use:

  flow   route_files on host files: the `-cap/-net/-out` run of the executable
         (read, pin selection, trees, routing, guides written).
  route  one Router.run() of an opened design, then what a program reads back:
         the routed demand of every layer and, with `score`, the device
         evaluator's totals.  Plain and batched forms, with and without the
         learned congestion seed, 1 to 3 rip-up-and-reroute passes.
  tree   one phase-1 batch on a grid context: the full cost refresh and the
         tree DP over the caller's device arrays.
  seed_predict / seed_grad / seed_train
         the learned congestion seed: tiled inference of a whole feature map,
         one forward and backward pass on given tiles, one optimiser step on
         random tiles of resident maps.

Designs come from the repository's own generator with the distributions of its
benchmark configurations (256x256 with blockages, 840x1140 with 65-500-pin
nets, 512x512 and 1600x1600 with the 2-1000-pin mixture and six hotspots).
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch
import torch.nn.functional as F

import instantgr_b200 as ig

# pin mixtures of the benchmark's designs: "blocked" = pin counts geometric, 5%
# of the edges in blockages; "fanout" = the same pins and 1% nets of 65-500
# pins; "mixed" = 2 to 1000 pins, six hotspots
MIXES = {
    "blocked": dict(cap_mode=0, block_frac=0.05, pin_mode=0, hifanout_frac=0.0, bbox_median=8.0, bbox_sigma=1.0,
                    hotspots=0, hotspot_frac=0.0),
    "fanout": dict(cap_mode=1, block_frac=0.0, pin_mode=0, hifanout_frac=0.01, bbox_median=8.0, bbox_sigma=1.0,
                   hotspots=0, hotspot_frac=0.0),
    "mixed": dict(cap_mode=1, block_frac=0.0, pin_mode=1, hifanout_frac=0.0, bbox_median=10.0, bbox_sigma=1.2,
                  hotspots=6, hotspot_frac=0.35),
}
NODES_PER_NET = {"blocked": 5.0, "fanout": 8.0, "mixed": 8.0}  # tree nodes, for work()

# the seed network: channels in and out, mode (0 same size, 1 stride 2, 2 nearest x2 first), ReLU
LAYERS = [(16, 32, 0, True), (32, 64, 1, True), (64, 64, 0, True), (64, 64, 0, True), (64, 32, 2, True),
          (32, 16, 0, False)]
OUT_LAYERS = 10
LR = 1e-3


def listed() -> list[dict]:
    return [
        # a whole command-line run on a small design: what one block of a floorplan costs
        dict(name="flow_20k", kind="flow", X=256, Y=256, nets=20000, mix="blocked", rrr=1),
        # a trial route of a few hundred nets, where launches and synchronisations count
        dict(name="route_300", kind="route", X=61, Y=44, nets=300, mix="blocked", rrr=1, batched=0, seeded=0, score=0),
        # a block routed with the batched form and the learned seed, the form tuned for quality per time
        dict(name="route_40k_seeded", kind="route", X=512, Y=512, nets=40000, mix="mixed", rrr=3, batched=1,
             seeded=1, score=0),
        # a mid-size design with high-fanout nets, routed and scored
        dict(name="route_130k", kind="route", X=840, Y=1140, nets=130000, mix="fanout", rrr=3, batched=0, seeded=0,
             score=1),
        # the benchmark's full-size design, routed and scored
        dict(name="route_800k", kind="route", X=1600, Y=1600, nets=800000, mix="mixed", rrr=3, batched=0, seeded=0,
             score=1),
        # phase-1 batches of a host that drives the loop itself: the last nets of a small grid ...
        dict(name="tree_64", kind="tree", X=200, Y=141, nets=64),
        # ... an ordinary batch of a mid-size grid ...
        dict(name="tree_6k", kind="tree", X=840, Y=1140, nets=6000),
        # ... and the largest batches of a full-size grid
        dict(name="tree_100k", kind="tree", X=1600, Y=1600, nets=100000),
        # congestion prediction for one small block (a single tile) and for a full-size design
        dict(name="predict_150", kind="seed_predict", X=150, Y=97),
        dict(name="predict_1600", kind="seed_predict", X=1600, Y=1600),
        # loss and gradients of a few given tiles: gradient checks and custom training loops
        dict(name="grad_2x64", kind="seed_grad", tiles=2, S=64, halo=16),
        # training as the shipped model was trained: one step of 16 tiles of 288 x 288
        dict(name="train_16x288", kind="seed_train", tiles=16, S=288, halo=16, maps=4, map_side=512),
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choice(["flow", "route", "route", "tree", "tree", "seed_predict", "seed_grad", "seed_train"])
    if kind in ("flow", "route"):
        nets = int(_log(rng, 300, 30000 if kind == "flow" else 400000))
        cells = nets / rng.uniform(0.1, 0.31)
        aspect = rng.uniform(0.6, 1.6)
        X = max(32, int(math.sqrt(cells * aspect)))
        Y = max(32, int(math.sqrt(cells / aspect)))
        side = min(X, Y)  # the wide nets of the other mixtures need room
        mix = rng.choice(["blocked"] if side < 150 else ["blocked", "mixed"] if side < 260 else list(MIXES))
        c = dict(kind=kind, X=X, Y=Y, nets=nets, mix=mix, rrr=rng.randint(1, 3))
        if kind == "route":
            c.update(batched=rng.randint(0, 1), seeded=rng.randint(0, 1), score=rng.randint(0, 1))
        return c
    if kind == "tree":
        cells = _log(rng, 3e4, 2.5e6)
        aspect = rng.uniform(0.6, 1.6)
        return dict(kind=kind, X=int(math.sqrt(cells * aspect)), Y=int(math.sqrt(cells / aspect)),
                    nets=int(_log(rng, 64, 100000)))
    if kind == "seed_predict":
        return dict(kind=kind, X=int(_log(rng, 60, 1600)), Y=int(_log(rng, 60, 1600)))
    halo = rng.choice([8, 12, 16])
    if kind == "seed_grad":
        return dict(kind=kind, tiles=rng.randint(1, 6), S=2 * rng.randint(halo + 4, 72), halo=halo)
    S = 2 * rng.randint(halo + 16, 144)
    return dict(kind=kind, tiles=rng.randint(1, 16), S=S, halo=halo, maps=rng.randint(1, 6),
                map_side=rng.randint(max(64, S - 2 * halo), 512))


# ------------------------------------------------------------------ inputs
def _design(case: dict, seed: int) -> dict:
    d = tempfile.TemporaryDirectory(prefix="igr_case_")
    cap, net = os.path.join(d.name, "d.cap"), os.path.join(d.name, "d.net")
    ig.generate_custom(case["X"], case["Y"], case["nets"], seed=seed % (1 << 40) + 1, cap=cap, net=net,
                       **MIXES[case["mix"]])
    return dict(dir=d, cap=cap, net=net)


def _trees(X: int, Y: int, n: int, r) -> tuple:
    """Batch of n trees in preorder: 2 to 200 nodes, mostly under 8; a child lies a short run from its parent,
    half of the edges bent; pins on layers 0 and 1, about a third of the inner nodes Steiner points (layer 9)."""
    u = r.random(n)
    cnt = np.where(u < 0.7, r.integers(2, 4, n), np.where(u < 0.9, r.integers(3, 9, n), r.integers(9, 21, n)))
    if n >= 400:
        big = r.random(n) < 0.002
        cnt = np.where(big, r.integers(33, 200, n), cnt)
    off = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    total = int(off[-1])
    net = np.repeat(np.arange(n), cnt)
    loc = np.arange(total) - off[net]
    # preorder parents: mostly the previous node, else an earlier one near it
    back = np.where(r.random(total) < 0.65, 1, r.integers(1, 5, total))
    par = np.where(loc == 0, -1, np.maximum(0, loc - back)).astype(np.int32)
    bent = r.random(total) < 0.5
    dx = np.rint(np.exp(r.normal(1.6, 0.9, total)) * np.where(r.random(total) < 0.5, 1, -1)).astype(np.int64)
    dy = np.rint(np.exp(r.normal(1.6, 0.9, total)) * np.where(r.random(total) < 0.5, 1, -1)).astype(np.int64)
    flat = r.random(total) < 0.5
    dx[~bent & flat] = 0
    dy[~bent & ~flat] = 0
    x, y = np.empty(total, np.int64), np.empty(total, np.int64)
    root = loc == 0
    x[root], y[root] = r.integers(0, X, n), r.integers(0, Y, n)
    for k in range(1, int(cnt.max())):  # one level of local indices at a time
        i = np.nonzero(loc == k)[0] if k < 8 else (off[:-1] + k)[cnt > k]
        p = off[net[i]] + par[i]
        x[i] = np.clip(x[p] + dx[i], 0, X - 1)
        y[i] = np.clip(y[p] + dy[i], 0, Y - 1)
    inner = np.zeros(total, bool)
    inner[(off[net] + np.maximum(par, 0))[loc > 0]] = True
    layer = r.integers(0, 2, total)
    layer[inner & ~root & (r.random(total) < 0.33)] = 9
    nodes = (layer * X * Y + x * Y + y).astype(np.int32)
    cap = (8 * cnt + 1).astype(np.int32)
    roff = np.concatenate([[0], np.cumsum(cap.astype(np.int64))[:-1]])
    return off.astype(np.int32), nodes, par, cap, roff.astype(np.int64), int(cap.sum())


def _grid(X: int, Y: int, r) -> "ig.Ctx":
    """Nine routing layers with the benchmark's integer capacities (means 10 to 4, +-2) under half-unit demand that
    fills most of them and overfills a few."""
    mean = np.linspace(10, 4, 9, dtype=np.float32)[:, None, None]
    cap = np.maximum(0, mean + r.integers(-2, 3, (9, X, Y), dtype=np.int32)).astype(np.float32)
    dem = (0.5 * r.integers(0, 22, (9, X, Y), dtype=np.int32)).astype(np.float32)
    c = ig.Ctx(9, X, Y, 0, r.integers(1, 3, X - 1), r.integers(1, 3, Y - 1), 1.0, 2.0, np.ones(9), cap)
    c.set_demand(dem)
    return c


def _features(X: int, Y: int, gen) -> torch.Tensor:
    """Channels-last features as a design's: pins per GCell, two smooth wire densities, blocked fraction, capacities;
    BF16 values, as the design path makes them."""
    dev = "cuda"
    f = torch.zeros(X, Y, 16, device=dev)
    f[..., 0] = 0.25 * torch.poisson(torch.full((X, Y), 1.4, device=dev), generator=gen)
    lo = torch.rand(2, 1, X // 16 + 2, Y // 16 + 2, device=dev, generator=gen) * 2.0
    f[..., 1:3] = F.interpolate(lo, size=(X, Y), mode="bilinear")[:, 0].permute(1, 2, 0)
    f[..., 3] = (torch.rand(X, Y, device=dev, generator=gen) < 0.03).float() / 9
    mean = torch.linspace(10, 4, 9, device=dev)
    f[..., 5:14] = (mean + torch.randint(-2, 3, (X, Y, 9), device=dev, generator=gen)).clamp_min(0) / 8
    return f.bfloat16().float()


def _targets(f: torch.Tensor, gen) -> torch.Tensor:
    """Demand maps that follow the wire densities, in half units of 1/8 track, layers 1 to 9."""
    t = torch.zeros_like(f)
    share = torch.linspace(1.4, 0.4, 9, device=f.device)
    base = torch.where((torch.arange(9, device=f.device) % 2 == 0), f[..., 1:2], f[..., 2:3]) * share
    noise = torch.rand(base.shape, device=f.device, generator=gen) * 2
    t[..., 1:10] = ((base * 4 + noise) * 2).round().clamp_min(0) / 16
    return t.bfloat16().float()


def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _tiles(case: dict, seed: int) -> tuple:
    g = _gen(seed)
    f = torch.stack([_features(case["S"], case["S"], g) for _ in range(case["tiles"])])
    return f.cpu().numpy(), torch.stack([_targets(t, g) for t in f]).cpu().numpy()


def _maps(case: dict, seed: int) -> list:
    g = _gen(seed)
    out = []
    for _ in range(case["maps"]):
        f = _features(case["map_side"], case["map_side"], g)
        out.append((f, _targets(f, g)))
    return out


def _model_params() -> np.ndarray:
    return np.load(ig.SEED_MODEL_PATH)["params"]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = dict(case=case)
    if kind == "flow":
        s.update(_design(case, seed))
        s["out"] = os.path.join(s["dir"].name, "d.out")
        s["guides"] = np.zeros(1024 * (case["nets"] + 1000), np.uint8)  # room for the guide file, zeros after its end
    elif kind == "route":
        d = _design(case, seed)
        r = ig.Router(d["cap"], d["net"], rrr_iters=case["rrr"], batched=case["batched"])
        if case["seeded"]:
            s["model"] = ig.Seed.load()
            r.set_seed(s["model"])
        s["router"] = r
        d["dir"].cleanup()
    elif kind == "tree":
        r = np.random.default_rng(seed)
        s["ctx"] = _grid(case["X"], case["Y"], r)
        off, nodes, par, cap, roff, total = _trees(case["X"], case["Y"], case["nets"], r)
        dev = {k: torch.from_numpy(v).cuda() for k, v in
               dict(off=off, nodes=nodes, par=par, cap=cap, roff=roff).items()}
        room = 64 * case["nets"] + 8192  # one pool of records for every batch of this size
        if total > room:
            raise RuntimeError("the records do not fit their pool")
        s.update(dev, room=room, stamp=0, nnodes=len(nodes), routes=torch.zeros(room, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
    elif kind == "seed_predict":
        s["model"] = ig.Seed.load()
        s["features"] = _features(case["X"], case["Y"], _gen(seed)).cpu().numpy()
    elif kind == "seed_grad":
        s["model"] = ig.Seed.load()
        s["model"].set_tile(case["S"], case["halo"])
        s["x"], s["t"] = _tiles(case, seed)
    else:
        m = s["model"] = ig.Seed.load()
        m.set_tile(case["S"], case["halo"])
        for f, t in _maps(case, seed):
            m.add_map(f.cpu().numpy(), t.cpu().numpy())
        s["calls"] = 0
    return s


def run(s: dict):
    case = s["case"]
    kind = case["kind"]
    if kind == "flow":
        ig.route_files(s["cap"], s["net"], s["out"], rrr_iters=case["rrr"])
        with open(s["out"], "rb") as f:
            f.readinto(s["guides"])
            if f.read(1):
                raise RuntimeError("the guide file is longer than its buffer")
        return s["guides"]
    if kind == "route":
        s["router"].run()
        out = dict(demand=s["router"].demand())
        if case["score"]:
            out["score"] = s["router"].evaluate()
        return out
    if kind == "tree":
        s["stamp"] += 1
        s["ctx"].cost_refresh()
        s["ctx"].pattern_route_static(case["nets"], s["off"].data_ptr(), s["nnodes"], s["nodes"].data_ptr(),
                                      s["par"].data_ptr(), s["roff"].data_ptr(), s["cap"].data_ptr(),
                                      s["routes"].data_ptr(), s["room"], s["stamp"])
        return s["routes"]
    if kind == "seed_predict":
        return s["model"].predict(s["features"])
    if kind == "seed_grad":
        loss, g = s["model"].grad(s["x"], s["t"])
        return dict(loss=loss, grads=g)
    s["calls"] += 1
    curve = s["model"].train(1, tiles=case["tiles"], lr=LR, seed=s["calls"])
    return dict(loss=curve.astype(np.float32), params=s["model"].params())


# ------------------------------------------------------------------ work
def _conv_flops(S: int) -> float:
    h = S // 2
    side = [S, h, h, h, S, S]
    return sum(2.0 * 9 * ci * co * n * n for (ci, co, _, _), n in zip(LAYERS, side))


def work(case: dict) -> dict:
    kind = case["kind"]
    params = sum(9 * ci * co + co for ci, co, _, _ in LAYERS)
    if kind in ("flow", "route", "tree"):
        cells = 9.0 * case["X"] * case["Y"]
        nodes = case["nets"] * NODES_PER_NET[case["mix"]] if kind != "tree" else case["nets"] * 6.0
        record = 4 * 9 * nodes  # a record's positions, 4 bytes each, about 9 per tree node
        if kind == "tree":  # capacity and demand in, two cost tables out; trees in, records out
            return dict(bytes=cells * (4 + 4 + 4 + 8) + 8 * nodes + record, flops=0)
        if kind == "flow":  # the two files in, the guide file out
            return dict(bytes=cells * 10 / 9 * 2.2 + nodes * 20 + nodes * 50, flops=0)
        return dict(bytes=cells * (4 + 4) + 8 * nodes + record, flops=0)  # capacity, trees in; demand, records out
    if kind == "seed_predict":
        px = float(case["X"] * case["Y"])
        return dict(bytes=px * 16 * (4 + 4) + 4 * params, flops=_conv_flops(288) / 288 ** 2 * px)
    px = float(case["tiles"] * case["S"] ** 2)
    fl = case["tiles"] * (3 * _conv_flops(case["S"]) - 2.0 * 9 * 16 * 32 * case["S"] ** 2)
    if kind == "seed_grad":
        return dict(bytes=px * 16 * (4 + 4) + 8 * params, flops=fl)
    return dict(bytes=px * 16 * (2 + 2) + 4 * 7 * params, flops=fl)  # tiles in BF16; weights, moments in and out


# ------------------------------------------------------------------ values in 64 bits
def _split(p: torch.Tensor) -> list:
    out, o = [], 0
    for ci, co, _, _ in LAYERS:
        w = p[o:o + 9 * ci * co].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        o += 9 * ci * co
        out.append((w, p[o:o + co]))
        o += co
    return out


def _network(x: torch.Tensor, p: torch.Tensor) -> torch.Tensor:
    """x [T][S][S'][16] -> [T][S][S'][16], in the type of its inputs."""
    a = x.permute(0, 3, 1, 2)
    for (w, b), (_, _, mode, relu) in zip(_split(p), LAYERS):
        if mode == 2:
            a = F.interpolate(a, scale_factor=2, mode="nearest")
        a = F.conv2d(a, w, b, stride=2 if mode == 1 else 1, padding=1)
        if relu:
            a = torch.relu(a)
    return a.permute(0, 2, 3, 1)


def _loss_and_grads(x: np.ndarray, t: np.ndarray, halo: int) -> tuple:
    p = torch.from_numpy(_model_params()).double().cuda().requires_grad_()
    loss, S = 0.0, x.shape[1]
    count = x.shape[0] * (S - 2 * halo) ** 2 * OUT_LAYERS
    for i in range(x.shape[0]):  # one tile at a time: the activations in 64 bits are large
        y = _network(torch.from_numpy(x[i:i + 1]).double().cuda(), p)
        e = (y - torch.from_numpy(t[i:i + 1]).double().cuda())[:, halo:S - halo, halo:S - halo, :OUT_LAYERS]
        part = (e * e).sum() / count
        part.backward()
        loss += part.item()
    return loss, p.grad, p.detach()


def _splitmix(state: int) -> tuple:
    m = (1 << 64) - 1
    state = (state + 0x9E3779B97F4A7C15) & m
    z = state
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return state, z ^ (z >> 31)


def _training_tiles(case: dict, seed: int) -> tuple:
    """The random tiles of the first training call: maps and corners from a splitmix64 stream, zeros outside a map."""
    maps = _maps(case, seed)
    S, halo, side = case["S"], case["halo"], case["map_side"]
    inner = S - 2 * halo
    state = (1 * 0x9E3779B97F4A7C15 + 3) & ((1 << 64) - 1)
    xs, ts = [], []
    for _ in range(case["tiles"]):
        state, v = _splitmix(state)
        f, t = maps[v % case["maps"]]
        at = [0, 0]
        if side > inner:
            for k in range(2):
                state, v = _splitmix(state)
                at[k] = v % (side - inner + 1)
        pad = S  # zeros on every side
        cut = [F.pad(m.permute(2, 0, 1), (pad, pad, pad, pad))[:, pad - halo + at[0]:pad - halo + at[0] + S,
                                                               pad - halo + at[1]:pad - halo + at[1] + S]
               for m in (f, t)]
        xs.append(cut[0].permute(1, 2, 0).contiguous().cpu().numpy())
        ts.append(cut[1].permute(1, 2, 0).contiguous().cpu().numpy())
    return np.stack(xs), np.stack(ts)


def exact(case: dict, seed: int):
    """Outputs in 64 bits: the seed network's.  Routes and demand are whole numbers (or half units) decided by the
    costs, with no value of their own in 64 bits."""
    kind = case["kind"]
    if kind == "seed_predict":
        X, Y, pad = case["X"], case["Y"], 16
        f = _features(X, Y, _gen(seed)).double()
        # outside the map the network sees zero features, as beyond a tile's edge: 16 GCells cover its reach
        f = F.pad(f.permute(2, 0, 1), (pad, pad + Y % 2, pad, pad + X % 2)).permute(1, 2, 0)[None]
        p = torch.from_numpy(_model_params()).double().cuda()
        out = np.empty((X, Y, 16))
        band = 256  # bands of rows with a margin: the activations in 64 bits are large
        with torch.no_grad():
            for x0 in range(0, X, band):
                y = _network(f[:, x0:x0 + band + 2 * pad + band % 2], p)[0, pad:pad + band, pad:pad + Y]
                k = min(band, X - x0)
                out[x0:x0 + k] = y[:k].cpu().numpy()
        return out
    if kind == "seed_grad":
        loss, g, _ = _loss_and_grads(*_tiles(case, seed), case["halo"])
        return dict(loss=loss, grads=g.cpu().numpy())
    if kind == "seed_train":
        loss, g, p = _loss_and_grads(*_training_tiles(case, seed), case["halo"])
        step = LR * g / (g.abs() + 1e-8)  # Adam's first step: both moments' corrections cancel
        return dict(loss=np.array([loss]), params=(p - step).cpu().numpy())
    return None
