"""What a user of this framework has it do, as cases that can be timed: single sparse layers, the 8-layer encoder in
inference and training, rule generation by itself, the voxeliser, and the conversions on either side of the path.

A case is a dict of plain values:
  kind      layer | encoder | rules | voxelize | sweep | coo
  B,H,W,D   scans and grid: H beams, W azimuth steps, D depth bins (the compressed axis)
  occ,nmax  share of the (h, w) columns that hold voxels, most voxels in a column
  depth     iid: depths drawn from the log-normal range distribution of the benchmark's configurations, independently;
            surface: neighbouring columns see the same surfaces, as in a sensor's sweep
  rules     what of the reference-format pair lists a pass produces: padded (the default settings: lists padded with -1),
            lists (the benchmark's setting: config.fill_unused_rules off), tables (config.materialize_rules off)
"""
import math

import torch

import sphconv_b200 as sphconv
from sphconv_b200 import quant, synthetic
from sphconv_b200 import sphconv_cuda as ops
from sphconv_b200.encoder import build_encoder8

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
ESIZE = {"fp32": 4, "fp16": 2, "bf16": 2, "int8": 1}
CART_RANGE, SPH_RANGE = [6, -40, -3, 70.4, 40, 1], [6, -45, 87.5, 70.4, 45, 100]
SCAN = dict(H=64, W=512, D=256, occ=0.9, nmax=4)        # the benchmark's scan


def listed():
    return [
        # the smallest call: one submanifold layer on one small scan (the benchmark's first configuration); its time is
        # launches and host work
        dict(name="layer_small", kind="layer", dtype="fp32", train=False, subm=True, ic=16, oc=16, kernel="3,3,3",
             stride="1,1,1", fused=False, rules="padded", depth="iid", B=1, H=32, W=128, D=64, occ=0.85, nmax=3),
        # one downsampling layer, forward and backward (the second configuration)
        dict(name="down_train", kind="layer", dtype="fp16", train=True, subm=False, ic=32, oc=64, kernel="3,3,3",
             stride="2,2,2", fused=False, rules="padded", depth="iid", B=4, H=64, W=512, D=128, occ=0.9, nmax=4),
        # a layer of channel counts that are no powers of two on a ragged grid, forward and backward
        dict(name="odd_train", kind="layer", dtype="fp16", train=True, subm=True, ic=24, oc=40, kernel="3,3,3",
             stride="1,1,1", fused=True, rules="padded", depth="surface", B=2, H=41, W=359, D=187, occ=0.8, nmax=4),
        # one scan at a time through the backbone: what an online detector waits for
        dict(name="encoder_1", kind="encoder", dtype="fp16", train=False, rules="tables", depth="surface", B=1, **SCAN),
        # a batch of scans (the third configuration, the benchmark's headline)
        dict(name="encoder_8", kind="encoder", dtype="fp16", train=False, rules="lists", depth="iid", B=8, **SCAN),
        # a training step's forward and backward (the fourth configuration)
        dict(name="train_bf16", kind="encoder", dtype="bf16", train=True, rules="lists", depth="iid", B=16, **SCAN),
        # the same by a program written for the reference: float32, default settings, a small batch
        dict(name="train_fp32", kind="encoder", dtype="fp32", train=True, rules="padded", depth="iid", B=2, **SCAN),
        # quantised inference on wide scans (the fifth configuration, one of four GPUs' share)
        dict(name="int8_wide", kind="encoder", dtype="int8", train=False, rules="lists", depth="iid",
             **dict(SCAN, B=16, W=2048)),
        # rule generation by itself, as a caller of the operators has it: both kinds, odd sizes, default settings
        dict(name="rules_odd", kind="rules", kernel="3,3,3", stride="2,2,2", rules="padded", depth="iid", B=3, H=37,
             W=301, D=101, occ=0.7, nmax=5),
        # raw points of a batch of sweeps to the encoder's input tensor
        dict(name="voxelize_8", kind="voxelize", B=8, H=64, W=512, D=256, points=120000),
        # one sweep from raw points through the encoder to the dense tensor a detection head reads
        dict(name="sweep_dense", kind="sweep", dtype="fp16", rules="tables", B=1, H=64, W=512, D=256, points=120000),
        # coordinates + features to the sparse tensor and on to the dense one, and the gradient back
        dict(name="coo_dense", kind="coo", dtype="fp16", c=64, B=8, H=16, W=128, D=64, fill=0.3),
    ]


def draw(rng):
    def between(lo, hi):                                  # over the logarithm, both ends included
        return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))

    def grid(columns):                                    # a scan's grid and how many scans of it stay within `columns`
        H, W, D = between(16, 64), between(64, 1024), between(32, 256)
        return dict(B=between(1, max(1, min(16, columns // (H * W)))), H=H, W=W, D=D, occ=round(rng.uniform(0.3, 0.95), 2),
                    nmax=rng.randint(1, 5), depth=rng.choice(["iid", "surface"]))

    kind = rng.choice(["layer", "layer", "layer", "encoder", "encoder", "encoder", "rules", "voxelize", "sweep", "coo"])
    rules = rng.choice(["padded", "lists", "tables"])
    if kind == "layer":
        subm = rng.random() < 0.6
        channel = lambda: rng.choice([4, 8, 16, 32, 64, rng.randint(3, 64)])  # noqa: E731
        return dict(kind=kind, dtype=rng.choice(["fp32", "fp16", "bf16"]), train=rng.random() < 0.6, subm=subm,
                    ic=channel(), oc=channel(), kernel=rng.choice(["3,3,3", "3,3,3", "3,3,1", "1,3,3", "5,3,3"]),
                    stride="1,1,1" if subm else rng.choice(["2,2,2", "2,2,2", "1,1,2", "2,2,1"]), fused=rng.random() < 0.5,
                    rules="padded" if rules == "padded" else "lists", **grid(65536))
    if kind == "encoder":
        dtype, train = rng.choice([("fp16", False), ("fp16", False), ("int8", False), ("fp32", False), ("bf16", True),
                                   ("fp16", True), ("fp32", True)])
        return dict(kind=kind, dtype=dtype, train=train, rules=rules, **grid(65536 if dtype == "fp32" else 262144))
    if kind == "rules":
        return dict(kind=kind, kernel=rng.choice(["3,3,3", "3,3,3", "5,3,3"]), stride=rng.choice(["2,2,2", "1,1,2", "2,2,1"]),
                    rules="padded", **grid(65536))
    if kind == "coo":
        g = dict(H=between(8, 32), W=between(32, 256), D=between(16, 64))
        return dict(kind=kind, dtype=rng.choice(["fp32", "fp16"]), c=rng.choice([4, 16, 32, 64, rng.randint(3, 64)]),
                    B=between(1, max(1, min(8, (1 << 20) // (g["H"] * g["W"] * g["D"])))), fill=round(rng.uniform(0.02, 0.5), 2), **g)
    g = dict(B=1 if kind == "sweep" else between(1, 8), H=between(32, 64), W=between(256, 512), D=between(64, 256),
             points=between(5000, 120000))
    return dict(kind=kind, **g, **(dict(dtype="fp16", rules="tables") if kind == "sweep" else {}))


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _triple(text):
    return [int(v) for v in text.split(",")]


def _scans(case, seed, B=None):
    """z_idx [NNZ], z_ptr [B,H,W] of a batch of scans.  Another seed turns the sensor by a few steps (the field of view
    ends inside the grid) and changes the scans' order: other inputs whose outputs have the same sizes."""
    gen = _generator(1)
    B, H, W, D, nmax = B or case["B"], case["H"], case["W"] - 16, case["D"], case["nmax"]
    dev = gen.device
    rand = lambda *s: torch.rand(*s, generator=gen, device=dev)  # noqa: E731
    if case["depth"] == "iid":
        r = torch.exp(math.log(20.0) + 0.6 * torch.randn(B, H, W, nmax, generator=gen, device=dev))
        r = torch.where(r < 80.0, r, 80.0 * rand(B, H, W, nmax))
        bins = torch.floor(r / 80.0 * D)
    else:  # a smooth range image of a few waves, and a handful of returns close behind the surface
        h = torch.arange(H, device=dev).view(1, 1, H, 1) / H
        w = torch.arange(W, device=dev).view(1, 1, 1, W) / W
        p = rand(B, 6, 4)
        freq = torch.tensor([1.0, 2.0, 4.0, 7.0, 11.0, 17.0], device=dev).view(1, 6, 1, 1)
        wave = (0.15 + 0.25 * p[..., 0]).view(B, 6, 1, 1) * torch.sin(
            6.2832 * (freq * w + p[..., 1].view(B, 6, 1, 1) + (2.0 * p[..., 2].view(B, 6, 1, 1) - 1.0) * h))
        r = torch.exp(math.log(20.0) + wave.sum(1) + 0.01 * torch.randn(B, H, W, generator=gen, device=dev))
        step = torch.floor(rand(B, H, W, nmax) * 3.0)
        step[..., 0] = 0.0
        bins = torch.floor(r / 80.0 * D).unsqueeze(-1) + step.cumsum(-1)
    bins = bins.clamp_(0, D - 1).long()
    count = torch.where(rand(B, H, W) < case["occ"], 1 + (rand(B, H, W) * nmax).long(), 0)
    keep = torch.arange(nmax, device=dev) < count.unsqueeze(-1)
    column = torch.arange(B * H * W, device=dev).view(B, H, W, 1)
    key = torch.unique((column * D + bins)[keep])            # a bin drawn twice counts once
    b, hw = key // (D * W * H), key // D % (H * W)
    b, h, w = (b + seed // 3) % B, hw // W, hw % W + 4 * (1 + seed % 3)
    key = (((b * H + h) * case["W"] + w) * D + key % D).sort()[0]
    per_column = torch.bincount(key // D, minlength=B * H * case["W"])
    return (key % D).int(), per_column.cumsum(0).int().view(B, H, case["W"])


def _points(case, seed, B=None):
    """float32 [N,4] points of B sweeps in azimuth order, and their spherical coordinates; some lie outside the grid.
    Another seed starts the sweeps elsewhere, changes their order and draws new intensities."""
    gen = _generator(1)
    B, n = B or case["B"], case["points"]
    rand = lambda: torch.rand(B, n, generator=gen, device=gen.device)  # noqa: E731
    r0, p0, t0, r1, p1, t1 = [float(v) for v in SPH_RANGE]
    phi = torch.deg2rad(p0 + (1.08 * rand().sort(1)[0] - 0.04) * (p1 - p0))
    theta = torch.deg2rad(t0 + (1.08 * rand() - 0.04) * (t1 - t0))
    r = torch.exp(math.log(3.0 * r0) + 0.7 * torch.randn(B, n, generator=gen, device=gen.device)).clamp(0.5 * r0, 1.1 * r1)
    xyz = torch.stack([r * torch.sin(theta) * torch.cos(phi), r * torch.sin(theta) * torch.sin(phi), r * torch.cos(theta),
                       torch.rand(B, n, generator=_generator(seed), device=gen.device)], -1)
    return xyz.roll((seed % B, seed * 7919 % n), (0, 1)).reshape(B * n, 4).float().contiguous(), (r, phi, theta)


def _generator_for(case):
    return sphconv.VoxelGenerator(CART_RANGE, SPH_RANGE, 2, 200000, [case["D"], case["W"], case["H"]], "spherical")


def _out_shape(case, shape):
    if case.get("subm"):
        return shape
    k, s = _triple(case["kernel"]), _triple(case["stride"])
    return [(n + 2 * (a // 2) - a) // b + 1 for n, a, b in zip(shape, k, s)]


def prepare(case, seed):
    """Everything a program holds before the call: the scans on the device, the network with its weights."""
    gen = _generator(seed)
    dev = gen.device
    kind = case["kind"]
    st = {"case": case, "B": case["B"], "shape": [case["H"], case["W"], case["D"]]}
    if kind in ("voxelize", "sweep"):
        st["points"], _ = _points(case, seed)
        st["scan_ptr"] = torch.arange(case["B"] + 1, dtype=torch.int32) * case["points"]
        st["voxels"] = _generator_for(case)
        if kind == "sweep":
            st["net"] = build_encoder8(dtype=DTYPES[case["dtype"]], device=dev, seed=seed % 100000).eval()
        return st
    if kind == "coo":
        cells = case["B"] * case["H"] * case["W"] * case["D"]
        at = torch.randperm(cells, generator=gen, device=dev)[: max(1, int(cells * case["fill"]))]
        left, cols = at, []
        for n in (case["D"], case["W"], case["H"]):
            cols.append(left % n)
            left = left // n
        st["indices"] = torch.stack([left] + cols[::-1], 1).int().contiguous()
        st["feature"] = torch.randn(at.numel(), case["c"], generator=gen, device=dev).to(DTYPES[case["dtype"]])
        st["grad"] = torch.randn(case["B"], case["c"], *st["shape"], generator=gen, device=dev).to(DTYPES[case["dtype"]])
        return st
    st["z_idx"], st["z_ptr"] = _scans(case, seed)
    if kind == "rules":
        return st
    nnz = st["z_idx"].numel()
    channels = case.get("ic", 4)
    feature = torch.randn(nnz, channels, generator=gen, device=dev)
    if case["dtype"] == "int8":
        z_idx, z_ptr = _scans(case, seed + 1, B=1)
        calib = torch.randn(z_idx.numel(), channels, generator=gen, device=dev)
        float_net = build_encoder8(dtype=torch.float32, device=dev, seed=seed % 100000).eval()
        st["net"] = quant.quantize_encoder(float_net, sphconv.SparseConvTensor(calib, st["shape"], 1, z_idx=z_idx, z_ptr=z_ptr))
        st["feature"] = st["net"].quantize_input(feature)
        return st
    dtype = DTYPES[case["dtype"]]
    st["feature"] = feature.to(dtype)
    if kind == "encoder":
        st["net"] = build_encoder8(dtype=dtype, device=dev, seed=seed % 100000)
        out_cells, out_channels = case["B"] * math.prod((n + 3) // 4 for n in st["shape"]), 64
    else:
        k, s = _triple(case["kernel"]), _triple(case["stride"])
        more = dict(bias=True, apply_bias=True, activation="relu") if case["fused"] else dict(bias=False)
        cls = sphconv.SubMConv3d if case["subm"] else sphconv.Conv3d
        more.update({} if case["subm"] else dict(stride=s, padding=[v // 2 for v in k]))
        net = cls(case["ic"], case["oc"], k, indice_key="k", **more)
        with torch.no_grad():
            net.weight.copy_(torch.as_tensor(synthetic.make_weight(k, case["ic"], case["oc"], seed)))
            if net.bias is not None:
                net.bias.fill_(0.05)
        st["net"] = net.to(dev).to(dtype)
        out_channels = case["oc"]
        out_cells = nnz if case["subm"] else min(case["B"] * math.prod(_out_shape(case, st["shape"])),
                                                 nnz * math.prod(-(-a // b) for a, b in zip(k, s)))
    st["net"].train(case["train"])
    if case["train"]:   # the gradient that comes down from the layers above; a pass takes its first rows
        st["grad"] = torch.randn(out_cells, out_channels, generator=gen, device=dev).to(dtype)
    return st


# ---- one pass -------------------------------------------------------------------------------------------------------

def _settings(case):
    """The process-wide switches a program sets once."""
    rules = case.get("rules", "padded")
    sphconv.config.fill_unused_rules = rules == "padded"
    sphconv.config.materialize_rules = rules != "tables"


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    _settings(case)
    if kind == "voxelize":
        t = st["voxels"].to_tensor(st["points"], st["scan_ptr"])
        return {"feature": t.feature, "z_idx": t.z_idx, "z_ptr": t.z_ptr}
    if kind == "sweep":
        with torch.no_grad():
            return st["net"](st["voxels"].to_tensor(st["points"], st["scan_ptr"], dtype=DTYPES[case["dtype"]])).dense()
    if kind == "coo":
        feature = st["feature"].detach().requires_grad_(True)
        dense = sphconv.SparseConvTensor(feature, st["shape"], st["B"], indices=st["indices"]).dense()
        dense.backward(st["grad"])
        return {"dense": dense.detach(), "d_feature": feature.grad}
    if kind == "rules":
        k, s, shape = _triple(case["kernel"]), _triple(case["stride"]), st["shape"]
        p = [v // 2 for v in k]
        a = ops.get_rules_subm(st["z_idx"], st["z_ptr"], st["B"], shape, shape, k, [1, 1, 1], p, [1, 1, 1], [2, 2])
        b = ops.get_rules(st["z_idx"], st["z_ptr"], st["B"], shape, _out_shape(case, shape), k, s, p, [1, 1, 1], [2, 2])
        return {"subm": a[2:], "strided": b}
    with torch.set_grad_enabled(case["train"]):
        feature = st["feature"].detach().requires_grad_(case["train"])
        x = sphconv.SparseConvTensor(feature, st["shape"], st["B"], z_idx=st["z_idx"], z_ptr=st["z_ptr"])
        y = st["net"](x)
    out = {"feature": y.feature.detach(), "z_idx": y.z_idx, "z_ptr": y.z_ptr}
    if case["train"]:
        for p in st["net"].parameters():
            p.grad = None
        y.feature.backward(st["grad"][: y.feature.shape[0]])
        out["d_feature"] = feature.grad
        out["d_parameters"] = [p.grad for p in st["net"].parameters()]
    if kind == "layer" and case["rules"] == "padded":
        out["rules"], out["rule_size"] = y.rule_cache["k"][2:4]
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def _count(occ, out_shape, kernel, stride, subm):
    """(pairs, occupied output cells as a mask) of one layer on one scan's occupancy [H,W,D]."""
    p = [v // 2 for v in kernel]
    padded = torch.zeros([n + 2 * a for n, a in zip(occ.shape, p)], dtype=torch.bool, device=occ.device)
    padded[tuple(slice(a, a + n) for n, a in zip(occ.shape, p))] = occ
    views = [padded[tuple(slice(o, o + s * (n - 1) + 1, s) for o, s, n in zip(off, stride, out_shape))]
             for off in ((i, j, l) for i in range(kernel[0]) for j in range(kernel[1]) for l in range(kernel[2]))]
    out = occ
    if not subm:
        out = views[0].clone()
        for v in views[1:]:
            out |= v
    return sum(int((v & out).sum()) for v in views), out


def _rule_bytes(case, n_in, in_shape, out_shape, kernel, stride, pairs):
    """Bytes of the reference-format lists of one rule set ([tiles, KV, 2, capacity] and their lengths)."""
    tiles, kv = -(-out_shape[0] // 2) * -(-out_shape[1] // 2), math.prod(kernel)
    if case["rules"] == "tables":
        return 0
    if case["rules"] == "lists":
        return 8 * pairs + 4 * tiles * kv
    window = (stride[0] + kernel[0]) * (stride[1] + kernel[1])
    capacity = int(window * n_in / (in_shape[0] * in_shape[1]) * 2 + 64) & -16
    return 4 * tiles * kv * (2 * capacity + 1)


def work(case):
    """Every input read once, every output written once, layer by layer; 2 operations per multiply-add.  The voxels and
    pairs are counted on one scan and multiplied by the number of scans."""
    kind, B = case["kind"], case["B"]
    shape = [case["H"], case["W"], case["D"]]
    columns = B * shape[0] * shape[1]
    if kind == "coo":
        cells, e = columns * shape[2], ESIZE[case["dtype"]]
        n = int(cells * case["fill"])
        return {"bytes": n * 16 + 2 * n * case["c"] * e + 2 * cells * case["c"] * e, "flops": 0}
    nbytes = flops = 0
    occ = torch.zeros(shape, dtype=torch.bool, device=_device())
    if kind in ("voxelize", "sweep"):
        _, coords = _points(case, 0, B=1)
        lo, hi = SPH_RANGE[:3], SPH_RANGE[3:]
        cell = [((v[0] if i == 0 else torch.rad2deg(v[0])) - lo[i]) / (hi[i] - lo[i]) * (case["D"], case["W"], case["H"])[i]
                for i, v in enumerate(coords)]
        cell = torch.stack(cell[::-1], 1).floor().long()
        fits = ((cell >= 0) & (cell < torch.tensor(shape, device=cell.device))).all(1)
        occ[tuple(cell[fits].t())] = True
        nbytes += 16 * case["points"] * B + 20 * B * int(occ.sum()) + 4 * columns
        if kind == "voxelize":
            return {"bytes": nbytes, "flops": 0}
    else:
        z_idx, z_ptr = _scans(case, 0, B=1)
        per_column = torch.diff(z_ptr.view(-1), prepend=z_ptr.new_zeros(1))
        column = torch.repeat_interleave(torch.arange(per_column.numel(), device=z_idx.device), per_column.long())
        occ.view(-1)[column * shape[2] + z_idx.long()] = True
    if kind in ("encoder", "sweep"):
        layers = [(subm, ic, oc, [3, 3, 3], [s, s, s], key) for subm, ic, oc, s, key in synthetic.ENCODER8]
    elif kind == "layer":
        layers = [(case["subm"], case["ic"], case["oc"], _triple(case["kernel"]), _triple(case["stride"]), None)]
    else:
        layers = [(True, 0, 0, _triple(case["kernel"]), [1, 1, 1], "subm"),
                  (False, 0, 0, _triple(case["kernel"]), _triple(case["stride"]), None)]
    e, train = ESIZE[case.get("dtype", "fp32")], case.get("train", False)
    seen = {}
    for subm, ic, oc, k, s, key in layers:
        grid = list(occ.shape)
        out_grid = _out_shape(dict(subm=subm, kernel="%d,%d,%d" % tuple(k), stride="%d,%d,%d" % tuple(s)), grid)
        n_in = B * int(occ.sum())
        if key is None or key not in seen:
            pairs, out = _count(occ, out_grid, k, s, subm)
            pairs, n_out = pairs * B, B * int(out.sum())
            nbytes += 4 * (n_in + B * grid[0] * grid[1]) + (0 if subm else 4 * (n_out + B * out_grid[0] * out_grid[1]))
            nbytes += _rule_bytes(case, n_in, grid, out_grid, k, s, pairs)
            seen[key] = pairs, out, n_out
        pairs, out, n_out = seen[key]
        rows, weight = n_in * ic + n_out * oc, math.prod(k) * ic * oc
        nbytes += e * (rows + weight) * (2 if train else 1)      # backward: the gradient in, the gradients out
        flops += 2 * pairs * ic * oc * (3 if train else 1)
        if kind != "rules":
            occ = out
    if kind == "sweep":
        nbytes += e * 64 * B * occ.numel()
    return {"bytes": int(nbytes), "flops": int(flops)}


def tolerance(case):
    """Index outputs are exact.  Features: what the data type gives when sums are taken in another order."""
    kind, dtype = case["kind"], case.get("dtype", "fp32")
    if kind in ("rules", "coo"):
        return "exact"
    if kind == "voxelize":
        return {"rel": 1e-6}
    # `max` in training: a pre-activation next to zero may fall on the other side, and its gradient comes or goes
    more = {"max": 0.5} if case.get("train") else {}
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2, "int8": 1e-3}[dtype], **more}
