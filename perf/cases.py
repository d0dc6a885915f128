"""The work whose speed this project watches: what a user's program does with the framework, through
its public entry points, from a single small layer to whole networks.

A case is a dict of plain values with a ``kind``:

* ``conv``      one sparse convolution (submanifold, strided or transposed), rulebook built or reused,
                inference or forward + backward;
* ``backbone``  inference of the VoxelNet-style encoder of the benchmark configurations;
* ``unet``      forward + backward of the sparse UNet of the benchmark configurations;
* ``pool``      sparse max / average pooling, rulebook, forward + backward;
* ``voxelize``  points to voxels.

All inputs are synthetic and made on the GPU from the seed.  The voxels of a case form one scene, which each
seed moves, deals to the samples of the batch and lists in an order of its own: so the number of output voxels
belongs to the case, while coordinates, row order, neighbour maps, features and weights are those of the seed.
"""

import math

import torch

import spconv_triton_b200.pytorch as sp
from spconv_triton_b200 import constants
from spconv_triton_b200.pytorch.utils import PointToVoxel

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32, "tf32": torch.float32}
SIZES = {"fp16": 2, "bf16": 2, "fp32": 4, "tf32": 4}
LIDAR_GRID = (41, 1600, 1408)
INDOOR_GRID = (512, 512, 64)
# the samples of a batch differ in size, as frames of a sensor do; the mean over any batch is close to 1
RAGGED = (1.0, 0.85, 1.15, 0.93, 1.07, 0.8, 1.2, 1.0)


def listed():
    return [
        # the smallest call in use: one layer in PyTorch's default dtype on 2 000 voxels, as unit tests, demos
        # and small-object networks make it; latency and launches are what counts
        conv("subm_fp32_c16_2k", "subm", "uniform", "cube64", 1, 2000, 16, 16, 3, "fp32", bias=True),
        # online perception: one LiDAR frame through the encoder
        dict(name="backbone_fp16_b1", kind="backbone", batch=1, voxels=20000, dtype="fp16"),
        # the headline workload: a batch of eight frames through the same encoder
        dict(name="backbone_fp16_b8", kind="backbone", batch=8, voxels=20000, dtype="fp16"),
        # the published single-layer comparison: wide submanifold layer whose neighbour map an earlier layer
        # of the network has built
        conv("subm_fp16_c256_cached", "subm", "lidar", "lidar", 1, 50000, 256, 256, 3, "fp16", cached=True),
        # the published up-sampling comparison: wide transposed layer, map built in the pass, TF32
        conv("up_tf32_c256", "up", "lidar", "lidar", 1, 50000, 256, 256, 3, "tf32"),
        # training of a down-sampling layer on a large batch (map, forward, both gradients)
        conv("down_fp16_64_128_train", "down", "lidar", "lidar", 4, 120000, 64, 128, 3, "fp16", train=True, bias=True),
        # training in PyTorch's default dtype with IEEE arithmetic, an odd number of voxels
        conv("subm_fp32_c64_train", "subm", "indoor", "indoor", 1, 100003, 64, 64, 3, "fp32", train=True, bias=True),
        # the stress configuration: 125 offsets, 256 channels, dense-ish blobs, pair-list rulebook; the largest
        conv("subm_k5_fp16_c256_train", "subm", "blob", "cube256", 1, 400000, 256, 256, 5, "fp16", train=True, bias=True),
        # a training step of the segmentation network (forward and every gradient) under autocast
        dict(name="unet_fp16_train_b2", kind="unet", batch=2, voxels=120000, base=32, dtype="fp16"),
        # pooling between stages, both kinds, trained
        dict(name="maxpool_k2s2_fp16_train", kind="pool", op="max", k=2, stride=2, scene="blob", grid="cube256", batch=2,
             voxels=400000, channels=256, dtype="fp16"),
        dict(name="avgpool_k3s1_fp16_train", kind="pool", op="avg", k=3, stride=1, scene="blob", grid="cube256", batch=1,
             voxels=300000, channels=256, dtype="fp16"),
        # the step before a detector: eight LiDAR sweeps, or one aggregated cloud, to voxels
        dict(name="voxelize_1200k", kind="voxelize", points=1200000, per_voxel=5, features=4),
    ]


def conv(name, layer, scene, grid, batch, voxels, cin, cout, k, dtype, train=False, cached=False, bias=False):
    return dict(name=name, kind="conv", layer=layer, scene=scene, grid=grid, batch=batch, voxels=voxels, cin=cin,
                cout=cout, k=k, dtype=dtype, train=train, cached=cached, bias=bias)


def draw(rng):
    kind = rng.choice(["conv"] * 5 + ["backbone"] * 2 + ["unet"] + ["pool"] * 2 + ["voxelize"] * 2)
    if kind == "conv":
        return _draw_conv(rng)
    if kind == "backbone":
        return dict(kind=kind, batch=rng.randint(1, 8), voxels=_log(rng, 2000, 24000), dtype=rng.choice(["fp16", "fp16", "bf16"]))
    if kind == "unet":
        return dict(kind=kind, batch=rng.randint(1, 2), voxels=_log(rng, 10000, 120000), base=rng.choice([16, 32]), dtype="fp16")
    if kind == "pool":
        op, k, stride = rng.choice([("max", 2, 2), ("max", 3, 2), ("avg", 2, 2), ("avg", 3, 1)])
        scene, grid = rng.choice([("blob", "cube256"), ("lidar", "lidar"), ("uniform", "cube64")])
        most = 300000 if k == 2 else 60000 if scene != "blob" else 150000
        voxels = _log(rng, 3000, min(most, 100000 if grid == "cube64" else most))
        return dict(kind=kind, op=op, k=k, stride=stride, scene=scene, grid=grid, batch=rng.randint(1, 2), voxels=voxels,
                    channels=rng.choice([16, 32, 64, 96, 128, 256]), dtype=rng.choice(["fp16", "bf16", "fp32"]))
    return dict(kind=kind, points=_log(rng, 20000, 1200000), per_voxel=rng.choice([1, 5, 10, 32]),
                features=rng.choice([3, 4, 5]))


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_conv(rng):
    layer = rng.choice(["subm", "subm", "down", "up"])
    if layer == "up":
        scene, grid, low, high = rng.choice([("lidar", "lidar", 1000, 50000), ("uniform", "cube64", 1000, 40000)])
    else:
        scene, grid, low, high = rng.choice([
            ("lidar", "lidar", 2000, 120000), ("indoor", "indoor", 5000, 120000), ("blob", "cube256", 5000, 300000),
            ("uniform", "cube64", 1000, 60000), ("uniform", "plane512", 2000, 60000), ("uniform", "hyper64", 5000, 50000)])
    k = 3 if layer != "subm" or grid in ("hyper64",) else rng.choice([3, 3, 3, 5])
    dtype = rng.choice(["fp16", "fp16", "fp16", "bf16", "bf16", "fp32", "tf32"])
    cin = rng.choice([4, 16, 32, 48, 64, 96, 128, 256])
    cout = rng.choice([16, 32, 48, 64, 96, 128, 256])
    cached = layer == "subm" and rng.random() < 0.4
    if cached:
        cin = cout
    train, batch = rng.random() < 0.5, rng.randint(1, 4)
    bias = train or rng.random() < 0.5  # the layers' default is a bias; inference often has it folded into a normalisation
    # no dearer than the largest listed case: bounded by the pairs that a voxel can have at most in the scene
    reach = {"lidar": 8, "indoor": 10, "blob": 14, "uniform": 8}[scene] * (3 if layer == "up" else 1) * (3 if k == 5 else 1)
    flops = 2.0 * reach * cin * cout * batch * (3 if train else 1)
    high = min(high, int((6e10 if dtype == "fp32" else 8e11) / flops))
    high = min(high, int(1.2e9 / (reach * max(cin, cout) * batch)))
    voxels = _log(rng, min(low, max(high, 500)), max(high, 500))
    case = conv("", layer, scene, grid, batch, voxels, cin, cout, k, dtype, train, cached, bias)
    del case["name"]
    return case


# ---- scenes: int32 [N, 1 + ndim] on the GPU, rows of a sample in random order -------------------------------


def _grid(case):
    return {"lidar": LIDAR_GRID, "indoor": INDOOR_GRID, "cube64": (64,) * 3, "cube256": (256,) * 3,
            "plane512": (512,) * 2, "hyper64": (64,) * 4}[case["grid"]]


def _counts(case):
    return [max(64, int(case["voxels"] * RAGGED[b % len(RAGGED)])) for b in range(case["batch"])]


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device=gen.device)


def _ints(gen, low, high, shape):
    return torch.randint(int(low), int(high), shape, generator=gen, device=gen.device)


def _uniform_cells(gen, n, grid):
    return torch.stack([_ints(gen, 0, g, (n,)) for g in grid], 1)


def _lidar_cells(gen, n, grid, clusters=200, sigma=8.0, ground=0.7):
    """70 % on a noisy ground plane, 30 % in Gaussian clusters."""
    dev, m = gen.device, int(n * ground)
    z = torch.clamp(torch.round(2 + torch.randn(m, generator=gen, device=dev)), 0, 4).long()
    plane = torch.stack([z, _ints(gen, 0, grid[1], (m,)), _ints(gen, 0, grid[2], (m,))], 1)
    # the clusters of a scene stay where they are when more cells are drawn
    centres = torch.stack([_ints(torch.Generator(dev).manual_seed(gen.initial_seed() + d), 0, g, (clusters,))
                           for d, g in enumerate(grid)], 1)
    off = torch.round(torch.randn(n - m, 3, generator=gen, device=dev) * sigma).long()
    lumps = centres[_ints(gen, 0, clusters, (n - m,))] + off
    return torch.cat([plane, torch.minimum(lumps.clamp(min=0), torch.tensor(grid, device=dev) - 1)])


def _indoor_cells(gen, grid):
    """The walls of a few axis-aligned boxes and a few tilted planes, every cell of them."""
    dev = gen.device
    draws = _rand(gen, 8, 8).tolist()
    parts = []
    for r in draws[:5]:
        low = [int(r[0] * (grid[0] - 64)), int(r[1] * (grid[1] - 64)), int(r[2] * max(grid[2] - 24, 1))]
        size = [48 + int(r[3] * 208), 48 + int(r[4] * 208), 12 + int(r[5] * (grid[2] // 2 - 12))]
        high = [min(a + s, g - 1) for a, s, g in zip(low, size, grid)]
        for d in range(3):
            for face in (low[d], high[d]):
                axes = [torch.tensor([face], device=dev) if a == d else torch.arange(low[a], high[a] + 1, device=dev)
                        for a in range(3)]
                parts.append(torch.cartesian_prod(*axes))
    x, y = torch.meshgrid(torch.arange(grid[0], device=dev), torch.arange(grid[1], device=dev), indexing="ij")
    for r in draws[5:]:
        z = torch.round((r[0] - 0.5) * 0.16 * (x - grid[0] / 2) + (r[1] - 0.5) * 0.16 * (y - grid[1] / 2) + (0.2 + 0.6 * r[2]) * grid[2])
        cells = torch.stack([x, y, z.long()], -1).reshape(-1, 3)
        parts.append(cells[(cells[:, 2] >= 0) & (cells[:, 2] < grid[2])])
    return torch.cat(parts)


def _blob_cells(gen, want, grid):
    """The cells of random solid balls, at least ``want`` of them."""
    side, dev = grid[0], gen.device
    filled = torch.zeros(grid, dtype=torch.bool, device=dev)
    draws = _rand(gen, 4096, 4).tolist()
    for i, r in enumerate(draws):
        rad = side // 32 + int(r[3] * (side // 10 - side // 32))
        c = [rad + int(v * (side - 2 * rad)) for v in r[:3]]
        ax = torch.arange(-rad, rad + 1, device=dev).square()
        ball = ax[:, None, None] + ax[None, :, None] + ax[None, None, :] <= rad * rad
        filled[tuple(slice(v - rad, v + rad + 1) for v in c)] |= ball
        if i % 8 == 7 and int(filled.sum()) >= want:
            break
    return filled.nonzero()


def _keys(cells, grid):
    key = torch.zeros(cells.shape[0], dtype=torch.int64, device=cells.device)
    for d, g in enumerate(grid):
        key = key * g + cells[:, d].long()
    return key


def _cells_of(key, grid):
    cols = []
    for g in reversed(grid):
        cols.append(key % g)
        key = torch.div(key, g, rounding_mode="floor")
    return torch.stack(cols[::-1], 1)


def _sample(case, grid, b, n):
    """The cells of sample b of a case's scene: n distinct keys in ``grid``."""
    gen = torch.Generator(_device()).manual_seed(31 * b + 7)
    key = torch.zeros(0, dtype=torch.int64, device=_device())
    while key.shape[0] < n:
        m = int((n - key.shape[0]) * 1.3) + 64
        if case["scene"] == "uniform":
            cells = _uniform_cells(gen, m, grid)
        elif case["scene"] == "lidar":
            cells = _lidar_cells(gen, m, grid)
        elif case["scene"] == "indoor":
            cells = _indoor_cells(gen, grid)
        else:
            cells = _blob_cells(gen, n / 0.3, grid)
        key = torch.cat([key, _keys(cells, grid)]).unique()
    return key[torch.randperm(key.shape[0], generator=gen, device=_device())[:n]]


def scene(case, seed):
    """Voxel coordinates of a batch.  The cells keep away from the sides of the grid (but not from the floor), and
    a seed moves every sample by whole strides of the deepest level, so that the output voxels stay as many."""
    grid, rows, counts = _grid(case), [], _counts(case)
    upright = {"lidar": 0, "indoor": 2}.get(case["scene"])
    margin = [0 if d == upright else g // 16 for d, g in enumerate(grid)]
    inner = tuple(g - 2 * m for g, m in zip(grid, margin))
    gen = torch.Generator(_device()).manual_seed(1009 * seed + 1)
    steps = (2 * _rand(gen, len(counts), len(grid)) - 1).tolist()
    for b in range(len(counts)):
        which = (b + seed) % len(counts)
        key = _sample(case, inner, which, counts[which])
        cells = _cells_of(key[torch.randperm(key.shape[0], generator=gen, device=_device())], inner)
        for d, m in enumerate(margin):
            step = 8 if m >= 16 else 2
            cells[:, d] += m + step * int(steps[b][d] * 0.75 * m / step)
        rows.append(torch.cat([torch.full_like(cells[:, :1], b), cells], 1))
    return torch.cat(rows).int()


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cloud(n):
    """n points around a sensor; a seed gives them another order and other intensities."""
    gen = torch.Generator(_device()).manual_seed(1)
    return torch.randn(n, 3, generator=gen, device=_device()) * torch.tensor([18.0, 18.0, 0.9], device=_device())


# ---- the programs ---------------------------------------------------------------------------------------------


def _fill(net, gen):
    """Random weights with activations of about unit size, and normalisation statistics of a trained network."""
    with torch.no_grad():
        for m in net.modules():
            if isinstance(m, torch.nn.BatchNorm1d):
                for t, scale, shift in ((m.weight, 0.1, 1.0), (m.bias, 0.1, 0.0), (m.running_mean, 0.1, 0.0)):
                    t.copy_(shift + scale * torch.randn(t.shape, generator=gen, device=t.device))
                m.running_var.copy_(0.5 + _rand(gen, m.num_features))
            elif hasattr(m, "weight_shape"):
                fan_in = math.prod(m.weight_shape[1:])
                m.weight.copy_(torch.randn(m.weight_shape, generator=gen, device=m.weight.device) * (2.0 / fan_in) ** 0.5)
                if m.bias is not None:
                    m.bias.copy_(0.1 * torch.randn(m.bias.shape, generator=gen, device=m.bias.device))
    return net


def _norm_act(layer, channels, act=torch.nn.ReLU):
    return [layer, torch.nn.BatchNorm1d(channels, eps=1e-3, momentum=0.01), act()]


def _backbone():
    mods = _norm_act(sp.SubMConv3d(4, 16, 3, padding=1, bias=False, indice_key="subm0"), 16)
    cin = 16
    for level, cout in enumerate((32, 64, 64), 1):
        mods += _norm_act(sp.SparseConv3d(cin, cout, 3, stride=2, padding=1, bias=False, indice_key="down%d" % level), cout)
        for _ in range(2):
            mods += _norm_act(sp.SubMConv3d(cout, cout, 3, padding=1, bias=False, indice_key="subm%d" % level), cout)
        cin = cout
    return sp.SparseSequential(*mods)


def _unet(base):
    # a smooth activation: gradients through ReLU are discontinuous in the rounding of the activations
    smooth, w = torch.nn.SiLU, [base, 2 * base, 4 * base, 8 * base]
    mods = _norm_act(sp.SubMConv3d(4, w[0], 3, padding=1, bias=False, indice_key="subm0"), w[0], smooth)
    for i in range(1, 4):
        mods += _norm_act(sp.SparseConv3d(w[i - 1], w[i], 3, stride=2, padding=1, bias=False, indice_key="down%d" % i), w[i], smooth)
        mods += _norm_act(sp.SubMConv3d(w[i], w[i], 3, padding=1, bias=False, indice_key="subm%d" % i), w[i], smooth)
    for i in range(3, 0, -1):
        mods += _norm_act(sp.SparseInverseConv3d(w[i], w[i - 1], 3, indice_key="down%d" % i, bias=False), w[i - 1], smooth)
        mods += _norm_act(sp.SubMConv3d(w[i - 1], w[i - 1], 3, padding=1, bias=False, indice_key="subm%d" % (i - 1)), w[i - 1], smooth)
    return sp.SparseSequential(*mods)


def _conv_layer(case, cin, key=None):
    ndim = len(_grid(case))
    if case["layer"] == "subm":
        cls = (sp.SubMConv1d, sp.SubMConv2d, sp.SubMConv3d, sp.SubMConv4d)[ndim - 1]
        return cls(cin, case["cout"], case["k"], padding=case["k"] // 2, bias=case["bias"], indice_key=key)
    kinds = {"down": (sp.SparseConv1d, sp.SparseConv2d, sp.SparseConv3d, sp.SparseConv4d),
             "up": (sp.SparseConvTranspose1d, sp.SparseConvTranspose2d, sp.SparseConvTranspose3d, sp.SparseConvTranspose4d)}
    return kinds[case["layer"]][ndim - 1](cin, case["cout"], case["k"], stride=2, padding=1, bias=case["bias"])


def prepare(case, seed):
    dev, gen = _device(), torch.Generator(_device()).manual_seed(seed)
    state = {"kind": case["kind"], "tf32": case.get("dtype") == "tf32"}
    if case["kind"] == "voxelize":
        n = case["points"]
        pts = _cloud(n)[torch.randperm(n, generator=gen, device=dev)]
        state["points"] = torch.cat([pts, _rand(gen, n, max(case["features"] - 3, 0))], 1).contiguous()
        state["op"] = PointToVoxel([0.16, 0.16, 0.2], [-35.2, -40.0, -3.0, 35.2, 40.0, 1.0], case["features"],
                                   max(1000, 2 * n // 3), case["per_voxel"], dev)
        return state
    if case["kind"] in ("backbone", "unet"):
        lidar = case["kind"] == "backbone"
        case = dict(case, scene="lidar" if lidar else "indoor", grid="lidar" if lidar else "indoor")
    dtype = DTYPES[case["dtype"]]
    state.update(indices=scene(case, seed), grid=list(_grid(case)), batch=case["batch"])
    n = state["indices"].shape[0]
    if case["kind"] == "backbone":
        state["features"] = _rand(gen, n, 4).to(dtype)
        state["net"] = _fill(_backbone().to(dev), gen).to(dtype).eval()
    elif case["kind"] == "unet":
        state["features"], state["autocast"] = _rand(gen, n, 4), dtype
        state["net"] = _fill(_unet(case["base"]).to(dev), gen).train()
        # what the loss hands back, scaled so that 16-bit gradients neither overflow nor vanish
        state["grad"] = (0.05 * torch.randn(n, case["base"], generator=gen, device=dev)).to(dtype)
    elif case["kind"] == "pool":
        cls = sp.SparseMaxPool3d if case["op"] == "max" else sp.SparseAvgPool3d
        state["net"] = cls(case["k"], case["stride"]).to(dev).train()
        state["features"] = torch.randn(n, case["channels"], generator=gen, device=dev).to(dtype).requires_grad_()
    else:
        state["train"] = case["train"]
        state["net"] = _fill(_conv_layer(case, case["cin"], "map").to(dev), gen).to(dtype).train(case["train"])
        feats = torch.randn(n, case["cin"], generator=gen, device=dev).to(dtype)
        state["features"] = feats.requires_grad_(case["train"])
        if case["cached"]:  # an earlier layer of the network has built the neighbour map
            constants.SPCONV_ALLOW_TF32 = state["tf32"]
            with torch.no_grad():
                first = _fill(_conv_layer(case, case["cin"], "map").to(dev), gen).to(dtype).train(case["train"])
                x = first(sp.SparseConvTensor(feats.detach(), state["indices"], state["grid"], state["batch"]))
            state["earlier"] = x.replace_feature(state["features"])
    return state


def run(state):
    if state["kind"] == "voxelize":
        return state["op"].generate_voxel_with_id(state["points"])
    constants.SPCONV_ALLOW_TF32 = state["tf32"]
    net, feats = state["net"], state["features"]
    x = state.get("earlier")
    if x is None:
        x = sp.SparseConvTensor(feats, state["indices"], state["grid"], state["batch"])
    if state["kind"] == "backbone" or state["kind"] == "conv" and not state["train"]:
        with torch.no_grad():
            y = net(x)
        return y.features, y.indices
    params = list(net.parameters())
    for p in params:
        p.grad = None
    feats.grad = None
    if state["kind"] == "unet":
        with torch.autocast("cuda", dtype=state["autocast"]):
            y = net(x)
    else:
        y = net(x)
    # without a loss of its own, the gradient of half the sum of squares
    y.features.backward(state.get("grad", y.features.detach()))
    return [y.features.detach(), y.indices, feats.grad] + [p.grad for p in params]


# ---- what a pass cannot do without ----------------------------------------------------------------------------


def _offsets(k, ndim):
    return torch.cartesian_prod(*[torch.arange(k)] * ndim).reshape(-1, ndim).tolist()


def _rulebook_size(indices, grid, layer, k, stride=2, pad=1):
    """(output coordinates, output grid, number of input-output pairs) of a layer with this voxel set."""
    ndim = len(grid)
    stride, pad = (1, k // 2) if layer == "subm" else (stride, pad)
    if layer == "subm":
        out_grid = list(grid)
    elif layer == "up":
        out_grid = [(g - 1) * stride - 2 * pad + k for g in grid]
    else:
        out_grid = [(g + 2 * pad - k) // stride + 1 for g in grid]
    batch = int(indices[:, 0].max()) + 1
    full = [batch] + out_grid
    lim = torch.tensor(out_grid, device=indices.device)
    own = _keys(indices, full).sort()[0] if layer == "subm" else None
    pairs, outs = 0, torch.zeros(0, dtype=torch.int64, device=indices.device)
    for off in _offsets(k, ndim):
        o = torch.tensor(off, device=indices.device)
        if layer == "up":
            at = indices[:, 1:].long() * stride - pad + o
            ok = torch.ones(at.shape[0], dtype=torch.bool, device=at.device)
        else:
            at = indices[:, 1:].long() + pad - o
            ok = (at % stride == 0).all(1)
            at = torch.div(at, stride, rounding_mode="floor")
        ok &= ((at >= 0) & (at < lim)).all(1)
        key = _keys(torch.cat([indices[ok, :1].long(), at[ok]], 1), full)
        if layer == "subm":
            hit = torch.searchsorted(own, key).clamp(max=own.shape[0] - 1)
            pairs += int((own[hit] == key).sum())
        else:
            pairs += key.shape[0]
            outs = torch.cat([outs, key]).unique()
    return (indices if layer == "subm" else _cells_of(outs, full).int()), out_grid, pairs


def work(case):
    kind = case["kind"]
    if kind == "voxelize":
        # points in; of the outputs the point-to-voxel map and the voxels that the points can fill
        n = case["points"]
        voxels = min(_expected_voxels(n), max(1000, 2 * n // 3))
        return {"bytes": n * case["features"] * 4 + n * 8 + voxels * (16 + case["per_voxel"] * case["features"] * 4), "flops": 0}
    if kind in ("backbone", "unet"):
        lidar = kind == "backbone"
        case = dict(case, scene="lidar" if lidar else "indoor", grid="lidar" if lidar else "indoor")
    e, idx, grid = SIZES[case["dtype"]], scene(case, 0), list(_grid(case))
    n, row = idx.shape[0], 4 * (len(grid) + 1)
    if kind == "conv":
        out, _, pairs = _rulebook_size(idx, grid, case["layer"], case["k"])
        m, w = out.shape[0], case["cin"] * case["cout"] * case["k"] ** len(grid)
        forward = n * row + (n * case["cin"] + m * case["cout"] + w) * e + (0 if case["layer"] == "subm" else m * row)
        if case["cached"]:  # no coordinates, but the neighbour map
            forward += 4 * pairs - n * row
        # backward reads the gradient, the features and the weights again, and writes two gradients
        backward = (m * case["cout"] + 2 * n * case["cin"] + 2 * w) * e if case["train"] else 0
        return {"bytes": forward + backward, "flops": 2.0 * pairs * case["cin"] * case["cout"] * (3 if case["train"] else 1)}
    if kind == "pool":
        out, _, pairs = _rulebook_size(idx, grid, "down", case["k"], case["stride"], 0)
        m = out.shape[0]
        values = n * (3 if case["op"] == "max" else 2) + m * (3 if case["op"] == "max" else 2)
        return {"bytes": n * row + m * row + values * case["channels"] * e, "flops": 2.0 * pairs * case["channels"]}
    flops, weights, m, first = 0.0, 0, n, True
    width = [16, 32, 64, 64] if kind == "backbone" else [case["base"] << i for i in range(4)]
    cells = idx
    for level in range(4):
        c = width[level]
        if level:
            out, grid, pairs = _rulebook_size(cells, grid, "down", 3)
            # the decoder's inverse layer multiplies the same pairs once more
            flops += 2.0 * pairs * width[level - 1] * c * (1 if kind == "backbone" else 2)
            weights += 27 * width[level - 1] * c * (1 if kind == "backbone" else 2)
            cells = out
        _, _, pairs = _rulebook_size(cells, grid, "subm", 3)
        layers = [(4, c)] if not level else [(c, c)] * (2 if kind == "backbone" else 1)
        if kind == "unet" and level < 3:
            layers = layers + [(c, c)]
        for a, b in layers:
            flops += 2.0 * pairs * a * b
            weights += 27 * a * b
    if kind == "backbone":
        return {"bytes": n * (row + 4 * e) + weights * e + cells.shape[0] * (row + width[3] * e), "flops": flops}
    # forward and two gradients; fp32 weights read, their gradients written
    return {"bytes": n * (row + 16) + n * width[0] * e + 8 * weights, "flops": 3 * flops}


def _expected_voxels(n):
    """Distinct cells that the points meet."""
    pts = _cloud(n)
    cell = torch.floor(pts / torch.tensor([0.16, 0.16, 0.2], device=_device())).long() + 2048
    inside = (pts[:, 0].abs() < 35.2) & (pts[:, 1].abs() < 40.0) & (pts[:, 2] > -3.0) & (pts[:, 2] < 1.0)
    return int(_keys(cell[inside], [4096] * 3).unique().shape[0])


def tolerance(case):
    kind, dtype = case["kind"], case.get("dtype")
    if kind == "voxelize":
        return "exact"  # copies of inputs and whole numbers
    if kind == "unet":
        # a chain of fourteen layers with rounding to 16 bits, batch statistics and activations between them, and back
        return {"rel": 1e-2, "max": 0.4}
    if kind == "backbone":
        return {"rel": 3e-3 if dtype == "fp16" else 2e-2}
    if dtype == "fp32":
        return {"rel": 1e-5, "max": 4e-4}
    if dtype == "tf32":
        return {"rel": 5e-4}  # operands rounded to TF32 before fp32 sums
    return {"rel": 2e-3 if dtype == "fp16" else 1e-2}
