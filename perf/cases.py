"""The work that users of this engine have it do, as measurable cases.

Every case is a dict of plain values.  ``listed()`` names the ones that are tracked, ``draw()`` gives more of the
same ranges, ``prepare()`` makes what a program has in hand before the call (inputs, modules, and kernel maps where
the program has run a layer on the tensor before), ``run()`` is one pass through the public operator surface.

The clouds follow the shapes the engine is benchmarked on (uniform grid sample, spinning-LiDAR scans, rooms and
grids of rooms voxelised at 2 cm), generated on the device.  Features are N(0, 1).
"""
from __future__ import annotations

import functools
import json
import math

import torch

import pcengine_b200 as pce
from pcengine_b200.backend import conv_fwd_d2_cuda, mapping_d2_cuda

DTYPES = {"fp16": torch.float16, "fp32": torch.float32}
CLASSES = 19
VOXEL = 0.05  # metres, LiDAR scans


def listed():
    return [
        # The smallest call: one 3x3x3 layer on a small cloud in fp32 (PyTorch's default type), map included.
        # Latency and launches are all there is.
        dict(name="layer_uniform_20k_c16_fp32", kind="layer", cloud="uniform", voxels=20000, cin=16, cout=16, ks=3,
             dtype="fp32", tag="D2", maps="fresh"),
        # A later layer of a network on an indoor scene: the map exists, only the convolution runs.
        dict(name="layer_room_200k_c64_fp16", kind="layer", cloud="rooms", rooms=1, voxels=200000, cin=64, cout=64, ks=3,
             dtype="fp16", tag="D2", maps="kept"),
        # The explicit gather -> GEMM -> scatter dataflow (tag D1), map included, on a sparse room.
        dict(name="layer_room_40k_c128_d1_fp16", kind="layer", cloud="rooms", rooms=1, voxels=40000, cin=128, cout=128, ks=3,
             dtype="fp16", tag="D1", maps="fresh"),
        # One resolution level of a U-Net a user writes out of conv3d layers: down, submanifold, up; maps built by the
        # layers that first need them.
        dict(name="level_lidar2_c32_64_fp16", kind="level", cloud="lidar", scans=2, voxels=60000, cin=32, cout=64, ks=2,
             dtype="fp16"),
        # A residual block out of conv3d / BatchNorm / ReLU modules and an addition, maps kept from earlier layers.
        dict(name="block_lidar4_c96_fp16", kind="block", cloud="lidar", scans=4, voxels=60000, cin=96, cout=96, ks=3,
             dtype="fp16"),
        # Online segmentation of one scan: latency of a whole network pass, maps included.
        dict(name="unet_lidar1_fp16", kind="unet", cloud="lidar", scans=1, voxels=60000, cr=1.0, dtype="fp16", stream=False),
        # Batched serving: the coordinates' arrival is an event, so a batch's maps may be built while the one before
        # it computes.
        dict(name="unet_lidar8_fp16", kind="unet", cloud="lidar", scans=8, voxels=60000, cr=1.0, dtype="fp16", stream=True),
        # The same network, half as wide, in fp32 on a sparse room.
        dict(name="unet_room_25k_fp32", kind="unet", cloud="rooms", rooms=1, voxels=25000, cr=0.5, dtype="fp32", stream=False),
        # A large scene: 20 rooms, 5x5x5 kernel, map included.
        dict(name="layer_scene_1500k_c64_ks5_fp16", kind="layer", cloud="rooms", rooms=20, voxels=1500000, cin=64, cout=64,
             ks=5, dtype="fp16", tag="D2", maps="fresh"),
        # The same scene through a wide layer with the map kept: the most arithmetic in one call.
        dict(name="layer_scene_1500k_c256_fp16", kind="layer", cloud="rooms", rooms=20, voxels=1500000, cin=256, cout=256,
             ks=3, dtype="fp16", tag="D2", maps="kept"),
        # The front end: raw points of a batch of scans to one collated voxel tensor.
        dict(name="voxelise_lidar8", kind="voxelise", cloud="lidar", scans=8, voxels=60000),
        # The backend functions called as the original Python layer calls them (map, pair lists, convolution).
        dict(name="backend_lidar1_c64_fp16", kind="backend", cloud="lidar", scans=1, voxels=60000, cin=64, cout=64, ks=3,
             dtype="fp16"),
    ]


# ---- drawing ---------------------------------------------------------------------------------------------------

_WIDTHS = (4, 16, 19, 32, 48, 64, 96, 128, 160, 192, 256)
_MOST_FLOPS = {"fp16": 4e11, "fp32": 2e10}  # estimated with 8 pairs per row: bounded by the largest listed cases


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_cloud(rng, most_voxels):
    cloud = rng.choice(("uniform", "lidar", "rooms", "rooms"))
    if cloud == "uniform":
        return dict(cloud="uniform", voxels=_log_int(rng, 2000, min(60000, most_voxels)))
    if cloud == "lidar":
        scans = rng.randint(1, max(1, min(8, most_voxels // 60000)))
        return dict(cloud="lidar", scans=scans, voxels=_log_int(rng, 8000, 64000))
    voxels = _log_int(rng, 5000, most_voxels)
    return dict(cloud="rooms", rooms=max(1, -(-voxels // 150000)), voxels=voxels)


def draw(rng):
    kind = rng.choice(("layer", "layer", "layer", "level", "block", "unet", "unet", "voxelise", "backend"))
    dtype = rng.choice(("fp16", "fp16", "fp16", "fp32"))
    if kind == "voxelise":
        return dict(kind=kind, cloud="lidar", scans=rng.randint(1, 8), voxels=_log_int(rng, 8000, 64000))
    if kind == "unet":
        cloud = _draw_cloud(rng, 400000 if dtype == "fp16" else 30000)
        if dtype == "fp32" and cloud["cloud"] == "lidar":
            cloud = dict(cloud="rooms", rooms=1, voxels=_log_int(rng, 5000, 30000))
        return dict(kind=kind, **cloud, cr=rng.choice((0.5, 1.0)) if dtype == "fp16" else 0.5, dtype=dtype,
                    stream=rng.random() < 0.5)
    cin, cout = rng.choice(_WIDTHS), rng.choice(_WIDTHS[1:])
    if kind in ("block", "backend"):
        cin = cout = rng.choice((32, 64, 96, 128))
    ks = rng.choice((3, 3, 3, 5)) if kind == "layer" else (rng.choice((2, 2, 3)) if kind == "level" else 3)
    pairs = 8 if ks < 5 else 16
    most = int(_MOST_FLOPS[dtype] / (2.0 * pairs * cin * cout * (3 if kind in ("level", "block") else 1)))
    most = max(5000, min(most, 1500000 if kind == "layer" else 300000))
    case = dict(kind=kind, **_draw_cloud(rng, most), cin=cin, cout=cout, ks=ks, dtype=dtype)
    if kind == "layer":
        tag = rng.choice(("D2", "D2", "auto", "D1" if case["voxels"] <= 60000 and ks == 3 else "D2"))
        case.update(tag=tag, maps=rng.choice(("fresh", "kept")))
    return case


# ---- clouds (int32 [N,4] = (b,x,y,z), on the device) -----------------------------------------------------------

def _gen(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _rand(g, *shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=g.device)


def _key(c):
    c = c.long()
    return ((c[..., 0] * 65536 + c[..., 1]) * 65536 + c[..., 2]) * 4096 + c[..., 3]


def _unkey(k):
    return torch.stack([k // (65536 * 65536 * 4096), k // (65536 * 4096) % 65536, k // 4096 % 65536, k % 4096], 1).int()


def _lidar_points(g, azimuths):
    """A 64-beam spinning scan in the order of the sweep: every ray hits the nearest of a ground plane and 40 boxes
    standing on it.  Rays that end within a hundredth of a voxel of a voxel's border are left out."""
    dev = g.device
    el = torch.deg2rad(torch.linspace(-25.0, 3.0, 64, device=dev))[None, :]
    az = (torch.arange(azimuths, device=dev) * (2 * math.pi / azimuths))[:, None]
    d = torch.stack([el.cos() * az.cos(), el.cos() * az.sin(), el.sin() + 0 * az], -1).reshape(-1, 3)
    t = torch.where(d[:, 2] < 0, -1.7 / d[:, 2], torch.inf)
    ang, rad = _rand(g, 40, hi=2 * math.pi), 50.0 * _rand(g, 40).sqrt()
    side = _rand(g, 40, 3, lo=0.5, hi=5.0)
    ctr = torch.stack([rad * ang.cos(), rad * ang.sin(), -1.7 + side[:, 2] / 2], 1)
    lo, hi = ctr - side / 2, ctr + side / 2
    t1, t2 = lo[None] / d[:, None], hi[None] / d[:, None]
    near, far = torch.minimum(t1, t2).amax(2), torch.maximum(t1, t2).amin(2)
    hit = (far >= near) & (near > 0)  # (a box around the sensor has near < 0: no hit)
    t = torch.minimum(t, torch.where(hit, near, torch.inf).amin(1))
    p = d * t[:, None] + torch.tensor([51.0, 51.0, 2.02], device=dev)
    frac = p / VOXEL - torch.floor(p / VOXEL)
    return p[(t <= 50.0) & (frac > 0.01).all(1) & (frac < 0.99).all(1)]


def _lidar_scan(g, voxels):
    """(points, first point of its voxel) of the leading sector of a scan that fills exactly ``voxels`` voxels; a scan
    that meets too few of them is taken again with denser azimuths."""
    azimuths = 64 + voxels // 26
    while True:
        p = _lidar_points(g, azimuths)
        key, at = torch.unique(_key(torch.floor(torch.cat([p[:, :1] * 0, p / VOXEL], 1))), return_inverse=True)
        if len(key) >= voxels:
            break
        azimuths = azimuths * 5 // 4
    index = torch.arange(len(p), device=g.device)
    first = torch.full_like(key, len(p)).scatter_reduce_(0, at, index, "amin")
    keep = first[at] <= torch.sort(first).values[voxels - 1]
    return p[keep], (first[at] == index)[keep]


def _room_points(g, rooms, n_points):
    """Area-uniform samples of the surfaces of 8x8x3 m rooms with 30 boxes each, five rooms to a row."""
    dev = g.device
    shell = torch.tensor([[[8.0, 8.0, 3.0]]], device=dev).expand(rooms, 1, 3)
    side = torch.cat([shell, _rand(g, rooms, 30, 3, lo=0.3, hi=2.0)], 1)
    room = torch.arange(rooms, device=dev)
    origin = torch.stack([(room % 5) * 8.0, torch.div(room, 5, rounding_mode="floor") * 8.0, room * 0.0], 1)
    floor = torch.tensor([1.0, 1.0, 0.0], device=dev)
    at = _rand(g, rooms, 31, 3) * (8.0 - side) * floor  # boxes stand on the floor
    at[:, 0] = 0.0
    area = torch.stack([side[..., 1] * side[..., 2], side[..., 0] * side[..., 2], side[..., 0] * side[..., 1]], 2)  # per axis
    face = torch.multinomial(area.repeat_interleave(2, 2).reshape(-1), n_points, replacement=True, generator=g)
    box, axis = torch.div(face, 6, rounding_mode="floor"), torch.div(face % 6, 2, rounding_mode="floor")
    u = _rand(g, n_points, 3)
    u.scatter_(1, axis[:, None], (face % 2)[:, None].float())
    p = at.reshape(-1, 3)[box] + u * side.reshape(-1, 3)[box] + origin[torch.div(box, 31, rounding_mode="floor")]
    return p + 1e-4


def _points(g, voxels):
    """Raw points of one scan: 1.5 per occupied voxel, as a sensor returns them."""
    p, first = _lidar_scan(g, voxels)
    more = torch.randint(len(p), (voxels // 2,), generator=g, device=g.device)
    index = torch.cat([torch.nonzero(first)[:, 0], more])
    return p[torch.sort(index).values]


def _cloud(case, g):
    if case["cloud"] == "uniform":
        lin = torch.randperm(64 ** 3, generator=g, device=g.device)[: case["voxels"]]
        return torch.stack([0 * lin, lin // 4096, lin // 64 % 64, lin % 64], 1).int()
    if case["cloud"] == "lidar":
        parts = []
        for b in range(case["scans"]):
            p, first = _lidar_scan(g, case["voxels"])
            parts.append(_key(torch.floor(torch.cat([p[first][:, :1] * 0 + b, p[first] / VOXEL], 1))))
        return _unkey(torch.sort(torch.cat(parts)).values)
    n, samples = case["voxels"], int(case["voxels"] * 1.15)
    while True:
        p = torch.floor(_room_points(g, case["rooms"], samples) / 0.02)
        key = torch.unique(_key(torch.cat([p[:, :1] * 0, p], 1)))
        if len(key) >= n:
            return _unkey(torch.sort(key[torch.randperm(len(key), generator=g, device=g.device)[:n]]).values)
        samples = samples * 6 // 5


# ---- preparing -------------------------------------------------------------------------------------------------

class _Level(torch.nn.Module):
    def __init__(self, cin, cout, ks):
        super().__init__()
        self.down, self.mid = pce.conv3d(cin, cout, ks, 2), pce.conv3d(cout, cout, 3, 1)
        self.up = pce.conv3d(cout, cin, ks, 2, transposed=True)

    def forward(self, x):
        y = self.mid(self.down(x))
        return y, self.up(y)


class _Block(torch.nn.Module):
    def __init__(self, c, ks):
        super().__init__()
        self.conv1, self.bn1 = pce.conv3d(c, c, ks, 1), pce.BatchNorm(c)
        self.conv2, self.bn2 = pce.conv3d(c, c, ks, 1), pce.BatchNorm(c)
        self.relu = pce.ReLU(True)

    def forward(self, x):
        y = self.relu(self.bn1(self.conv1(x)))
        return self.relu(self.bn2(self.conv2(y)) + x)


def _tensor(s):
    return pce.spTensor(s["feats"], s["coords"], None, [0, 0, 0], s["cmax"], batchsize=s["batch"], init_tag=list(s["tags"]))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = _gen(seed, dev)
    kind = case["kind"]
    if kind == "voxelise":
        points = [_points(g, case["voxels"]) for _ in range(case["scans"])]
        return dict(kind=kind, points=points, feats=[torch.randn(len(p), 4, generator=g, device=dev) for p in points])
    dtype = DTYPES[case["dtype"]]
    coords = _cloud(case, g)
    cin = 4 if kind == "unet" else case["cin"]
    s = dict(kind=kind, coords=coords, feats=torch.randn(len(coords), cin, generator=g, device=dev).to(dtype),
             cmax=coords[:, 1:].amax(0).tolist(), batch=case.get("scans", 1), tags=["auto"])
    if kind == "backend":
        kv = case["ks"] ** 3
        w = torch.randn(kv, cin, case["cout"], generator=g, device=dev) / math.sqrt(kv * cin)
        s.update(ks=case["ks"], kernel=w.to(dtype))
        return s
    torch.manual_seed(seed)
    with torch.device(dev):
        if kind == "layer":
            net = pce.conv3d(cin, case["cout"], case["ks"], 1)
            s.update(tags=[case["tag"], "end"])
        elif kind == "level":
            net = _Level(cin, case["cout"], case["ks"])
        elif kind == "block":
            net = _Block(cin, case["ks"])
        else:
            net = pce.MinkUNet(4, CLASSES, case["cr"])
    pce.randomize_batchnorm(net, seed)
    s["net"] = net.to(dtype).eval()
    if case.get("stream"):
        s["ready"] = torch.cuda.Event()
        s["ready"].record()
    if case.get("maps") == "kept" or kind == "block":
        s["x"] = _tensor(s)
        with torch.no_grad():
            s["net"](s["x"])  # the layer before this one: it left its map on the tensor
    return s


# ---- one pass --------------------------------------------------------------------------------------------------

def _code(v):
    return 94273 * v + 311 * v + v


def _run_backend(s):
    coords, feats, kernel, ks = s["coords"], s["feats"], s["kernel"], s["ks"]
    n, kv, dev = len(coords), ks ** 3, coords.device
    imap = -torch.ones(kv * n, dtype=torch.int, device=dev)
    knnz = torch.zeros(kv, dtype=torch.int, device=dev)
    kpos = torch.zeros(kv + 1, dtype=torch.int, device=dev)
    qkpos = torch.zeros(kv + 1, dtype=torch.int, device=dev)
    mapping_d2_cuda(coords, s["batch"], _code(ks), kv, kernel.size(1), kernel.size(2), _code(1), _code(1), _code(0), 0, 0, 0,
                    *s["cmax"], imap, knnz, kpos, qkpos, True)
    nonzero_idx = torch.nonzero(imap != -1)
    omap = imap[nonzero_idx]
    imap = (nonzero_idx % n).int()
    sum_nnz = qkpos[-1].cpu().int()
    out = torch.zeros((n, kernel.size(2)), dtype=feats.dtype, device=dev)
    conv_fwd_d2_cuda(feats, kernel, _code(ks), sum_nnz, out, kpos, qkpos, imap, omap, True, True)
    return dict(feats=out, kpos=kpos)


def _run_voxelise(s):
    samples, inverse = [], []
    for points, feats in zip(s["points"], s["feats"]):
        voxels, index, inv = pce.sparse_quantize(points, VOXEL, return_index=True, return_inverse=True)
        samples.append(pce.spTensor(feats[index], voxels, coords_max=[0, 0, 0]))
        inverse.append(inv)
    batch = pce.sparse_collate(samples)
    return dict(coords=batch.coords, feats=batch.feats, inverse=inverse)


def run(state):
    kind = state["kind"]
    with torch.no_grad():
        if kind == "voxelise":
            return _run_voxelise(state)
        if kind == "backend":
            return _run_backend(state)
        x = state["x"] if "x" in state else _tensor(state)
        if "ready" in state:
            x.coords_ready = state["ready"]
        if kind == "level":
            mid, up = state["net"](x)
            return up.feats  # (made of every value of `mid`)
        return state["net"](x).feats


# ---- what a pass cannot do without -----------------------------------------------------------------------------

def _pairs(coords, ks):
    """(row, offset) pairs of a submanifold map, the centre included."""
    key, _ = torch.sort(_key(coords + torch.tensor([0, 4, 4, 4], dtype=torch.int32, device=coords.device)))
    r, total = ks // 2, 0
    for dx in range(-r, r + 1):
        for dy in range(-r, r + 1):
            for dz in range(-r, r + 1):
                want = key + (dx * 65536 + dy) * 4096 + dz
                at = torch.searchsorted(key, want).clamp_(max=len(key) - 1)
                total += int((key[at] == want).sum())
    return total


def _coarser(coords, ks):
    """(coarser coordinates, pairs) of a stride-2 layer with kernel size 2 or 3."""
    c, outs, pairs = coords.long(), [], 0
    for o in range(ks ** 3):
        d = c.clone()
        d[:, 1:] -= torch.tensor([o // (ks * ks), o // ks % ks, o % ks], device=c.device)
        d = d[(d[:, 1:] % 2 == 0).all(1) & (d[:, 1:] >= 0).all(1)]
        d[:, 1:] = torch.div(d[:, 1:], 2, rounding_mode="floor")
        pairs += len(d)
        outs.append(_key(d))
    return _unkey(torch.unique(torch.cat(outs))), pairs


@functools.lru_cache(maxsize=64)
def _work(text):
    case = json.loads(text)
    dev = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")
    kind = case["kind"]
    coords = _cloud(case, _gen(0, dev))
    n = len(coords)
    if kind == "voxelise":
        # points in, the voxel of each out; coordinates out, feature rows (of one point per voxel) in and out
        return dict(bytes=float((12 + 8) * (n + n // 2) + (16 + 16 + 16) * n), flops=0.0)
    e = 2 if case["dtype"] == "fp16" else 4
    if kind in ("layer", "backend", "block"):
        cin, cout, kv, pairs = case["cin"], case["cout"], case["ks"] ** 3, _pairs(coords, case["ks"])
        fresh = case.get("maps") == "fresh" or kind == "backend"
        layers = 2 if kind == "block" else 1
        index = 16 * n if fresh else 4 * pairs
        return dict(bytes=float(e * (n * (cin + cout) + layers * kv * cin * cout) + index), flops=2.0 * layers * pairs * cin * cout)
    if kind == "level":
        cin, cout, ks = case["cin"], case["cout"], case["ks"]
        low, pairs = _coarser(coords, ks)
        flops = 2.0 * (2 * pairs * cin * cout + _pairs(low, 3) * cout * cout)
        weights = (2 * ks ** 3 * cin + 27 * cout) * cout
        return dict(bytes=float(16 * n + 16 * len(low) + e * (2 * n * cin + len(low) * cout + weights)), flops=flops)
    rows, p3, down = [n], [_pairs(coords, 3)], []
    for _ in range(4):
        coords, p = _coarser(coords, 2)
        rows.append(len(coords))
        p3.append(_pairs(coords, 3))
        down.append(p)
    cs = [int(case["cr"] * c) for c in (32, 32, 64, 128, 256, 256, 128, 96, 96)]
    layers = [(p3[0], 27, 4, cs[0]), (p3[0], 27, cs[0], cs[0]), (n, 1, cs[8], CLASSES)]

    def block(level, cin, cout):
        layers.extend([(p3[level], 27, cin, cout), (p3[level], 27, cout, cout)])
        if cin != cout:
            layers.append((rows[level], 1, cin, cout))

    for i in range(4):
        layers.append((down[i], 8, cs[i], cs[i]))
        block(i + 1, cs[i], cs[i + 1])
        block(i + 1, cs[i + 1], cs[i + 1])
        layers.append((down[3 - i], 8, cs[4 + i], cs[5 + i]))
        block(3 - i, cs[5 + i] + cs[3 - i], cs[5 + i])
        block(3 - i, cs[5 + i], cs[5 + i])
    weights = sum(kv * cin * cout for _, kv, cin, cout in layers)
    return dict(bytes=float(16 * n + e * (n * (4 + CLASSES) + weights)),
                flops=sum(2.0 * pairs * cin * cout for pairs, _, cin, cout in layers))


def work(case):
    return dict(_work(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)))


def tolerance(case):
    if case["kind"] == "voxelise":
        return "exact"  # whole numbers, and features copied row by row
    if case["dtype"] == "fp32":
        return {"rel": 2e-5 if case["kind"] == "unet" else 1e-5}  # another order of 32-bit sums
    # fp16 values, fp32 sums: the rounding of every layer's output (and of the products in the explicit dataflow)
    return {"rel": {"unet": 5e-3, "block": 2e-3, "level": 2e-3}.get(case["kind"], 1e-3)}
