"""Workloads of the sparse convolution path, for timing it and for comparing its results.

Each case is a plain dict.  prepare(case, seed) makes what a program has in hand before the
call (voxel grids, features, layers with their weights), run(state) makes one pass through the
public API, exact(case, seed) computes the same outputs in 64 bits with plain torch, and
work(case) counts the bytes and operations that the pass cannot do without.

Grids are sphere shells (depth-sensor-like surfaces), faces of boxes (buildings), random
scattered voxels or dense blocks.  A pass starts from a grid without a kernel map, as an
inference request or a training step on a new sample does: maps, coarse grids and everything
derived from them are part of the pass.
"""

from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvdb-core_gb300"))

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
DEV = "cuda"


def listed():
    return [
        # one FP32 layer on a grid of a few thousand leaves: latency and launches decide
        {"name": "layer_small_f32", "kind": "layer", "geometry": "random", "voxels": 20000, "side": 64, "cin": 16,
         "cout": 16, "precision": "f32"},
        # a batch of many small objects, half precision, channel counts that are no power of two,
        # batch norm in inference mode: conv -> norm -> ReLU -> strided conv
        {"name": "infer_ragged_f16", "kind": "infer", "geometry": "shells", "grids": 32, "shells": 1, "res_lo": 16,
         "res_hi": 64, "cin": 24, "cmid": 40, "cout": 40, "dtype": "f16", "norm": True},
        # the benchmark's step: four scans of 256^3, conv 3^3 -> ReLU -> conv 2^3 stride 2
        {"name": "infer_bf16", "kind": "infer", "geometry": "shells", "grids": 4, "shells": 3, "res_lo": 256,
         "res_hi": 256, "cin": 32, "cmid": 64, "cout": 64, "dtype": "bf16", "norm": False},
        # a wide layer on a large scan in FP8 (inference)
        {"name": "layer_wide_fp8", "kind": "layer", "geometry": "shells", "grids": 1, "shells": 3, "res_lo": 1024,
         "res_hi": 1024, "cin": 128, "cout": 256, "precision": "fp8"},
        # the decoder's step: transposed 2^3 stride-2 convolution back onto the finer grid
        {"name": "up_bf16", "kind": "up", "geometry": "shells", "grids": 1, "shells": 3, "res_lo": 512, "res_hi": 512,
         "cin": 256, "cout": 128, "dtype": "bf16"},
        # training step of a conv -> ReLU -> conv block, forward and backward
        {"name": "train_bf16", "kind": "train", "geometry": "boxes", "grids": 1, "boxes": 8, "res_lo": 512,
         "res_hi": 512, "cin": 64, "cmid": 64, "cout": 64, "dtype": "bf16"},
        {"name": "train_f32", "kind": "train", "geometry": "shells", "grids": 2, "shells": 2, "res_lo": 128,
         "res_hi": 160, "cin": 32, "cmid": 64, "cout": 32, "dtype": "f32"},
        # point clouds to grids and their 3^3 kernel map (the data side of every step)
        {"name": "points_to_map", "kind": "points", "geometry": "shells", "grids": 4, "shells": 3, "res_lo": 256,
         "res_hi": 256, "kernel": 3},
        # encoder / decoder neighbours of the convolutions: pooling and upsampling, with gradients
        {"name": "pool_bf16", "kind": "pool", "geometry": "shells", "grids": 4, "shells": 3, "res_lo": 256,
         "res_hi": 256, "cin": 64, "dtype": "bf16", "mode": "max"},
        # normalisation between convolutions, forward and backward
        {"name": "groupnorm_bf16", "kind": "groupnorm", "geometry": "shells", "grids": 4, "shells": 3, "res_lo": 256,
         "res_hi": 256, "cin": 64, "groups": 8, "dtype": "bf16"},
        # one served request from host memory to host memory: grid build and a four-layer stack
        {"name": "serve_bf16", "kind": "serve", "geometry": "shells", "grids": 1, "shells": 3, "res_lo": 256,
         "res_hi": 256, "cin": 32, "cmid": 64, "cout": 32, "dtype": "bf16"},
        # the map-free convolution on a dense block, forward and backward
        {"name": "halo_bf16", "kind": "halo", "geometry": "dense", "side": 96, "cin": 32, "cout": 64,
         "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "infer", "infer", "up", "train", "train", "points", "pool", "groupnorm",
                       "serve", "halo"])
    chans = [16, 24, 32, 48, 64, 96, 128]
    if kind == "halo":
        return {"kind": kind, "geometry": "dense", "side": _log_int(rng, 20, 96), "cin": rng.choice([16, 24, 32, 48]),
                "cout": rng.choice([16, 32, 40, 64]), "dtype": rng.choice(["bf16", "f32"])}
    res = _log_int(rng, 40, 400)
    c = {"kind": kind, "geometry": "shells", "grids": rng.randint(1, 6), "shells": rng.randint(1, 3),
         "res_lo": max(16, int(res * rng.uniform(0.4, 1.0))), "res_hi": res}
    if kind == "layer":
        c["precision"] = rng.choice(["f32", "fp8", "bf16"])
        c["cin"] = rng.choice([32, 64, 128] if c["precision"] == "fp8" else chans)
        c["cout"] = rng.choice([32, 64, 96, 128, 256])
        if rng.random() < 0.4:
            side = _log_int(rng, 24, 128)
            c = {"kind": kind, "geometry": "random", "voxels": max(50, int(side**3 * rng.uniform(0.03, 0.2))),
                 "side": side, "precision": c["precision"], "cin": c["cin"], "cout": c["cout"]}
    elif kind == "infer":
        c.update(cin=rng.choice(chans), cmid=rng.choice(chans), cout=rng.choice(chans),
                 dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), norm=rng.random() < 0.5)
    elif kind == "up":
        c.update(cin=rng.choice([64, 128, 256]), cout=rng.choice([32, 64, 128]),
                 dtype=rng.choice(["bf16", "bf16", "f32"]))
    elif kind == "train":
        if rng.random() < 0.5:
            del c["shells"]
            c.update(geometry="boxes", boxes=rng.randint(2, 8))
        c.update(cin=rng.choice([32, 64, 128]), cmid=rng.choice([32, 64, 96, 128]), cout=rng.choice([16, 32, 64, 128]),
                 dtype=rng.choice(["bf16", "bf16", "f32"]))
    elif kind == "points":
        c.update(kernel=rng.choice([2, 3, 3]))
    elif kind == "pool":
        c.update(cin=rng.choice(chans), dtype=rng.choice(["bf16", "f32", "f16"]), mode=rng.choice(["max", "avg"]))
    elif kind == "groupnorm":
        c.update(cin=rng.choice([16, 32, 48, 64, 96, 128]), groups=rng.choice([4, 8, 16]),
                 dtype=rng.choice(["bf16", "f32"]))
    elif kind == "serve":
        c.update(grids=1, cin=32, cmid=64, cout=32, dtype="bf16")
    # no drawn case costs more than the largest listed one: wide layers get smaller grids
    most = 0.15e12 if "f32" in (c.get("dtype"), c.get("precision")) else 0.3e12
    while work(c)["flops"] > most and c["geometry"] != "random":
        c["res_hi"] = max(16, int(c["res_hi"] * 0.8))
        c["res_lo"] = min(c["res_lo"], c["res_hi"])
    return c


# ------------------------------------------------------------------ geometry ------------
def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1009 + salt)


def _key(b, ijk):
    """Sort key of the grids' voxel order for coordinates in [0, 4096): the grid, then the upper
    node child (bits 11..7 of x, y, z), the lower node child (6..3) and the leaf voxel (2..0)."""
    x, y, z = ijk.long().unbind(-1)
    up = ((x >> 7) << 10) | ((y >> 7) << 5) | (z >> 7)
    lw = (((x >> 3) & 15) << 8) | (((y >> 3) & 15) << 4) | ((z >> 3) & 15)
    lf = ((x & 7) << 6) | ((y & 7) << 3) | (z & 7)
    return (b.long() << 36) | (up << 21) | (lw << 9) | lf


def _unkey(k):
    up, lw, lf = (k >> 21) & 0x7FFF, (k >> 9) & 0xFFF, k & 0x1FF
    x = ((up >> 10) << 7) | ((lw >> 8) << 3) | (lf >> 6)
    y = (((up >> 5) & 31) << 7) | (((lw >> 4) & 15) << 3) | ((lf >> 3) & 7)
    z = ((up & 31) << 7) | ((lw & 15) << 3) | (lf & 7)
    return k >> 36, torch.stack([x, y, z], -1).int()


def _resolutions(case):
    """One resolution per grid, spread over [res_lo, res_hi] on a logarithmic scale, in mixed order."""
    n, lo, hi = case["grids"], case["res_lo"], case["res_hi"]
    r = [int(round(lo * (hi / lo) ** ((i + 0.5) / n))) for i in range(n)]
    return [r[i] for i in torch.randperm(n, generator=torch.Generator().manual_seed(n)).tolist()]


# The shapes of a case's grids belong to the case, so that its outputs have the same sizes for
# every seed; the seed places them: an axis order, mirrored axes and an even shift, which give
# other leaves, another voxel order and other maps, and the same voxel counts on both levels.
def _place(ijk, seed):
    g = torch.Generator().manual_seed(int(seed) * 7919 + 5)
    ijk = ijk.long()[:, torch.randperm(3, generator=g).to(DEV)]
    flip = torch.randint(0, 2, (3,), generator=g).to(DEV)
    shift = 2 * torch.randint(0, 32, (3,), generator=g).to(DEV)
    return torch.where(flip == 1, 1151 - ijk, ijk) + shift


def _shell_points(case):
    """Voxels hit by points drawn on a union of sphere shells per grid (10 R^2 points per shell, so
    most voxels are hit several times), the grid of each, and the points per grid."""
    res = torch.tensor(_resolutions(case), device=DEV)
    n, s = res.numel(), case["shells"]
    g = _gen(n * 16 + s, 1)
    centres = 0.3 + 0.4 * torch.rand(n, s, 3, generator=g, device=DEV)
    radii = 0.2 + 0.25 * torch.rand(n, s, generator=g, device=DEV)
    count = 10 * s * res * res
    b = torch.repeat_interleave(torch.arange(n, device=DEV), count)
    cum = (radii**2).cumsum(1)
    u = torch.rand(b.numel(), generator=g, device=DEV) * cum[b, -1]
    which = (u[:, None] > cum[b]).sum(1).clamp(max=s - 1)
    d = torch.randn(b.numel(), 3, generator=g, device=DEV)
    p = centres[b, which] + radii[b, which][:, None] * (d / d.norm(dim=1, keepdim=True).clamp_min(1e-12))
    return b, torch.floor(p.clamp(0.0, 1.0 - 1e-6) * res[b][:, None] + 0.5).long(), res, count


def _box_voxels(case):
    """Voxels on the faces of random boxes per grid, with repeats, and the grid of each."""
    bs, vox = [], []
    for b, res in enumerate(_resolutions(case)):
        g = torch.Generator().manual_seed(200 + b)
        for _ in range(case["boxes"]):
            side = 0.1 + 0.4 * torch.rand(3, generator=g)
            lo = torch.rand(3, generator=g) * (1 - side)
            a, e = torch.floor(lo * res).long().tolist(), torch.floor((lo + side) * res).long().tolist()
            for axis in range(3):
                u, v = [t for t in range(3) if t != axis]
                gu, gv = torch.meshgrid(torch.arange(a[u], e[u] + 1, device=DEV),
                                        torch.arange(a[v], e[v] + 1, device=DEV), indexing="ij")
                for face in (a[axis], e[axis]):
                    pts = torch.empty(gu.numel(), 3, dtype=torch.long, device=DEV)
                    pts[:, axis] = face
                    pts[:, u] = gu.reshape(-1)
                    pts[:, v] = gv.reshape(-1)
                    vox.append(pts)
                    bs.append(torch.full_like(pts[:, 0], b))
    return torch.cat(bs), torch.cat(vox)


def _voxel_keys(case, seed):
    """Sorted keys of the case's voxels and their number of grids."""
    if case["geometry"] == "dense":
        r = torch.arange(case["side"], device=DEV)
        ijk = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
        return torch.sort(_key(torch.zeros_like(ijk[:, 0]), ijk)).values, 1
    if case["geometry"] == "random":
        s = case["side"]
        idx = torch.randperm(s**3, generator=_gen(seed, 1), device=DEV)[: case["voxels"]]
        ijk = torch.stack([idx // (s * s), idx // s % s, idx % s], 1)
        return torch.sort(_key(torch.zeros_like(idx), ijk)).values, 1
    b, ijk = _box_voxels(case) if case["geometry"] == "boxes" else _shell_points(case)[:2]
    return torch.unique(_key(b, _place(ijk, seed))), case["grids"]


def _jagged(case, seed):
    """(grid of each voxel, ijk, offsets) in the grids' voxel order."""
    keys, n = _voxel_keys(case, seed)
    b, ijk = _unkey(keys)
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.bincount(b, minlength=n).cumsum(0)
    return b, ijk, off


def _grid(case, seed):
    import fvdb

    _, ijk, off = _jagged(case, seed)
    return fvdb.GridBatch.from_ijk(fvdb.JaggedTensor.from_data_and_offsets(ijk, off))


def _dtype(case):
    p = case.get("dtype") or case["precision"]
    return torch.bfloat16 if p == "fp8" else DTYPES[p]


def _randn(seed, salt, shape, dtype):
    return torch.randn(shape, generator=_gen(seed, salt), device=DEV).to(dtype)


def _weights(case, seed):
    """Weights and biases of the case's layers, by name, in the case's data type: Kaiming-normal
    weights, small biases; batch-norm scales near one."""
    dt, w = _dtype(case), {}

    def conv(name, cout, cin, k, transposed=False, salt=0):
        fan = cin * (k**3 if not transposed else 1)
        shape = (cin, cout, k, k, k) if transposed else (cout, cin, k, k, k)
        w[name] = (_randn(seed, 100 + salt, shape, torch.float32) * math.sqrt(2.0 / fan)).to(dt)
        w[name + "_bias"] = (_randn(seed, 150 + salt, (cout,), torch.float32) * 0.1).to(dt)

    if case["kind"] == "layer":
        conv("w1", case["cout"], case["cin"], 3)
    elif case["kind"] == "up":
        conv("w1", case["cout"], case["cin"], 2, transposed=True)
    elif case["kind"] in ("infer", "train"):
        conv("w1", case["cmid"], case["cin"], 3)
        conv("w2", case["cout"], case["cmid"], 2 if case["kind"] == "infer" else 3, salt=1)
        if case.get("norm"):
            c = case["cmid"]
            w["mean"] = (_randn(seed, 201, (c,), torch.float32) * 0.2).to(dt)
            w["var"] = (1 + 0.3 * torch.rand(c, generator=_gen(seed, 202), device=DEV)).to(dt)
            w["gamma"] = (1 + _randn(seed, 203, (c,), torch.float32) * 0.1).to(dt)
            w["beta"] = (_randn(seed, 204, (c,), torch.float32) * 0.1).to(dt)
    elif case["kind"] == "groupnorm":
        c = case["cin"]
        w["gamma"] = (1 + _randn(seed, 203, (c,), torch.float32) * 0.1).to(dt)
        w["beta"] = (_randn(seed, 204, (c,), torch.float32) * 0.1).to(dt)
    elif case["kind"] == "halo":
        w["w1"] = (_randn(seed, 100, (case["cout"], case["cin"], 3, 3, 3), torch.float32)
                   * math.sqrt(2.0 / (27 * case["cin"]))).to(dt)
    elif case["kind"] == "serve":
        ch = [case["cin"], case["cmid"], case["cmid"], case["cout"]]
        for i, (a, b) in enumerate(zip(ch[:-1], ch[1:])):
            w["w%d" % i] = (_randn(seed, 100 + i, (b, a, 3, 3, 3), torch.float32) * math.sqrt(2.0 / (27 * a))).to(dt)
    return w


# ------------------------------------------------------------------ passes --------------
def _load_conv(layer, w, name):
    with torch.no_grad():
        layer.weight.copy_(w[name])
        layer.bias.copy_(w[name + "_bias"])


def prepare(case, seed):
    import fvdb

    kind, dt = case["kind"], None if case["kind"] == "points" else _dtype(case)
    st = {"case": dict(case)}
    if kind == "points":
        b, ijk, res, count = _shell_points(case)
        jitter = torch.rand(ijk.shape, generator=_gen(seed, 3), device=DEV) * 0.9 - 0.45
        p = (_place(ijk, seed) + jitter) / res[b][:, None]
        off = torch.zeros(case["grids"] + 1, dtype=torch.int64, device=DEV)
        off[1:] = count.cumsum(0)
        st["points"] = fvdb.JaggedTensor.from_data_and_offsets(p.float(), off)
        st["voxel_sizes"] = [[1.0 / r] * 3 for r in res.tolist()]
        return st
    w = _weights(case, seed)
    if kind == "serve":
        from fvdb.serving import ConvStack, Request

        _, ijk, _ = _jagged(case, seed)
        perm = torch.randperm(ijk.shape[0], generator=_gen(seed, 3), device=DEV)
        x = _randn(seed, 2, (ijk.shape[0], case["cin"]), dt)
        st["request"] = Request(rid=0, ijk=ijk[perm].cpu().pin_memory(), features=x[perm].cpu().pin_memory())
        model = ConvStack([case["cin"], case["cmid"], case["cmid"], case["cout"]], DEV, dtype=dt, seed=int(seed))
        model.weights = [w["w%d" % i] for i in range(3)]
        st["model"] = model
        return st
    grid = st["grid"] = _grid(case, seed)
    n = grid.total_voxels
    if kind == "layer":
        layer = fvdb.nn.SparseConv3d(case["cin"], case["cout"], 3).to(DEV, dt).eval()
        if case["precision"] == "fp8":
            layer.precision = "fp8"
        _load_conv(layer, w, "w1")
        st["net"] = layer
        st["x"] = _randn(seed, 2, (n, case["cin"]), dt)
    elif kind == "infer":
        mods = [fvdb.nn.SparseConv3d(case["cin"], case["cmid"], 3)]
        if case["norm"]:
            mods.append(fvdb.nn.BatchNorm(case["cmid"]))
        mods += [fvdb.nn.ReLU(), fvdb.nn.SparseConv3d(case["cmid"], case["cout"], 2, stride=2)]
        net = fvdb.nn.Sequential(*mods).to(DEV, dt).eval()
        _load_conv(net[0], w, "w1")
        _load_conv(net[-1], w, "w2")
        if case["norm"]:
            with torch.no_grad():
                net[1].running_mean.copy_(w["mean"])
                net[1].running_var.copy_(w["var"])
                net[1].weight.copy_(w["gamma"])
                net[1].bias.copy_(w["beta"])
        st["net"] = net
        st["x"] = _randn(seed, 2, (n, case["cin"]), dt)
    elif kind == "up":
        coarse = st["coarse"] = grid.conv_grid(2, 2)
        st["net"] = fvdb.nn.SparseConv3d(case["cin"], case["cout"], 2, stride=2, transposed=True).to(DEV, dt).eval()
        _load_conv(st["net"], w, "w1")
        st["x"] = _randn(seed, 2, (coarse.total_voxels, case["cin"]), dt)
    elif kind == "train":
        net = fvdb.nn.Sequential(fvdb.nn.SparseConv3d(case["cin"], case["cmid"], 3), fvdb.nn.ReLU(),
                                 fvdb.nn.SparseConv3d(case["cmid"], case["cout"], 3)).to(DEV, dt).train()
        _load_conv(net[0], w, "w1")
        _load_conv(net[2], w, "w2")
        st["net"] = net
        st["x"] = _randn(seed, 2, (n, case["cin"]), dt).requires_grad_(True)
        st["dy"] = _randn(seed, 4, (n, case["cout"]), dt)
    elif kind == "pool":
        st["x"] = _randn(seed, 2, (n, case["cin"]), dt).requires_grad_(True)
        st["dy"] = _randn(seed, 4, (n, case["cin"]), dt)
    elif kind == "groupnorm":
        net = fvdb.nn.GroupNorm(case["groups"], case["cin"]).to(DEV, dt).train()
        with torch.no_grad():
            net.weight.copy_(w["gamma"])
            net.bias.copy_(w["beta"])
        st["net"] = net
        st["x"] = (_randn(seed, 2, (n, case["cin"]), torch.float32) * 1.5 + 0.5).to(dt).requires_grad_(True)
        st["dy"] = _randn(seed, 4, (n, case["cin"]), dt)
    elif kind == "halo":
        st["w"] = w["w1"].requires_grad_(True)
        st["x"] = _randn(seed, 2, (n, case["cin"]), dt).requires_grad_(True)
        st["dy"] = _randn(seed, 4, (n, case["cout"]), dt)
    return st


def run(st):
    import fvdb

    case = st["case"]
    kind = case["kind"]
    if kind == "points":
        grid = fvdb.GridBatch.from_points(st["points"], st["voxel_sizes"])
        pack, _ = grid.sparse_conv_kernel_map(case["kernel"], 1)
        pack.build_implicit_gemm()
        return {"ijk": grid.ijk.jdata, "offsets": grid.joffsets, "map": pack.out_in_map[: grid.total_voxels]}
    if kind == "serve":
        from fvdb.serving import run_alone

        y, ijk = run_alone(st["model"], st["request"], DEV)
        return {"y": y, "ijk": ijk}
    grid = st["grid"]
    if kind in ("layer", "infer", "up"):
        with torch.no_grad():
            if kind == "up":
                out = st["net"](fvdb.nn.VDBTensor(st["coarse"], st["x"]), grid)
            else:
                out = st["net"](fvdb.nn.VDBTensor(grid, st["x"]))
        return {"y": out.data.jdata}
    x = st["x"]
    if kind == "train":
        net = st["net"]
        y = net(fvdb.nn.VDBTensor(grid, x)).data.jdata
        g = torch.autograd.grad(y, [x, net[0].weight, net[0].bias, net[2].weight, net[2].bias], st["dy"])
        return {"y": y.detach(), "dx": g[0], "dw1": g[1], "db1": g[2], "dw2": g[3], "db2": g[4]}
    if kind == "pool":
        pool = grid.max_pool if case["mode"] == "max" else grid.avg_pool
        low, coarse = pool(2, grid.jagged_like(x))
        up, _ = coarse.subdivide(2, low, fine_grid=grid)
        (dx,) = torch.autograd.grad(up.jdata, [x], st["dy"])
        return {"low": low.jdata.detach(), "up": up.jdata.detach(), "dx": dx}
    if kind == "groupnorm":
        net = st["net"]
        y = net(fvdb.nn.VDBTensor(grid, x)).data.jdata
        g = torch.autograd.grad(y, [x, net.weight, net.bias], st["dy"])
        return {"y": y.detach(), "dx": g[0], "dgamma": g[1], "dbeta": g[2]}
    y = grid.sparse_conv_halo(grid.jagged_like(x), st["w"]).jdata
    g = torch.autograd.grad(y, [x, st["w"]], st["dy"])
    return {"y": y.detach(), "dx": g[0], "dw": g[1]}


# ------------------------------------------------------------------ counts --------------
def _expected(case):
    """Expected voxels, neighbours per voxel of a 3^3 map, and voxels after coarsening by 2."""
    if case["geometry"] == "dense":
        n = case["side"]
        return n**3, (3 - 2 / n) ** 3, ((n + 1) // 2) ** 3
    if case["geometry"] == "random":
        dens = case["voxels"] / case["side"] ** 3
        return case["voxels"], 1 + 26 * dens, case["voxels"] * (1 - (1 - dens) ** 8) / (8 * dens)
    per = 0.605 * case["boxes"] if case["geometry"] == "boxes" else 1.37 * case["shells"]
    lo, hi, n = case["res_lo"], case["res_hi"], case["grids"]
    vox = sum(per * (lo * (hi / lo) ** ((i + 0.5) / n)) ** 2 for i in range(n))
    return vox, (9.4 if case["geometry"] == "boxes" else 13.1), vox * 0.27


def work(case):
    """Each input and weight read once, each output written once; one multiply and one add per
    (present neighbour, input channel, output channel)."""
    n, nb, nc = _expected(case)
    e = {"f32": 4, "bf16": 2, "f16": 2, "fp8": 2}[case.get("dtype") or case.get("precision") or "f32"]
    k = case["kind"]
    if k == "points":
        pts = sum(10 * case["shells"] * r * r for r in _resolutions(case))
        return {"bytes": pts * 12 + n * 12 + n * 4 * case["kernel"] ** 3, "flops": 0}
    ci, co = case["cin"], case.get("cout", case["cin"])
    if k == "layer":
        return {"bytes": n * (ci + co) * e + 27 * ci * co * e, "flops": 2 * n * nb * ci * co}
    if k == "infer":
        m = case["cmid"]
        return {"bytes": (n * ci + nc * co) * e + (27 * ci * m + 8 * m * co) * e,
                "flops": 2 * n * nb * ci * m + 2 * n * m * co}
    if k == "up":
        return {"bytes": (nc * ci + n * co) * e + 8 * ci * co * e, "flops": 2 * n * ci * co}
    if k == "train":
        m = case["cmid"]
        return {"bytes": n * (2 * ci + 2 * co) * e + 27 * 2 * (ci * m + m * co) * e,
                "flops": 6 * n * nb * (ci * m + m * co)}
    if k == "pool":
        return {"bytes": (n * ci * 4 + nc * ci) * e, "flops": 8 * n * ci}
    if k == "groupnorm":
        return {"bytes": n * ci * 4 * e, "flops": 16 * n * ci}
    if k == "serve":
        m = case["cmid"]
        return {"bytes": n * (12 + ci * e + co * e + 12), "flops": 2 * n * nb * (ci * m + m * m + m * co)}
    return {"bytes": n * (2 * ci + 2 * co) * e + 27 * 2 * ci * co * e, "flops": 6 * n * nb * ci * co}


# ------------------------------------------------------------------ 64 bits -------------
def _lookup(keys, b, ijk):
    """Row of each coordinate of grid b in the sorted keys, -1 where absent."""
    ok = ((ijk >= 0) & (ijk < 4096)).all(1)
    q = _key(b, ijk.clamp(0, 4095))
    at = torch.searchsorted(keys, q).clamp(max=keys.numel() - 1)
    return torch.where(ok & (keys[at] == q), at, -1)


class _Conv64(torch.autograd.Function):
    """y[t] = sum over offsets k of x[row(t, k)] W[k], offset by offset (rows: a list of index
    tensors, -1 = absent; W: [K, Cin, Cout])."""

    @staticmethod
    def forward(ctx, x, w, rows):
        y = x.new_zeros(rows[0].numel(), w.shape[2])
        for k, r in enumerate(rows):
            t = torch.nonzero(r >= 0).squeeze(1)
            y.index_add_(0, t, x[r[t]] @ w[k])
        ctx.save_for_backward(x, w)
        ctx.rows = rows
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dx, dw = torch.zeros_like(x), torch.zeros_like(w)
        for k, r in enumerate(ctx.rows):
            t = torch.nonzero(r >= 0).squeeze(1)
            dx.index_add_(0, r[t], dy[t] @ w[k].t())
            dw[k] = x[r[t]].t() @ dy[t]
        return dx, dw, None


def _rows3(keys):
    """Neighbour rows of every voxel for the 3^3 offsets, weight dimension 2 fastest."""
    b, ijk = _unkey(keys)
    return [_lookup(keys, b, ijk + torch.tensor([i, j, k], device=DEV, dtype=torch.int32))
            for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]


def _coarse(keys):
    """Keys of the coarse voxels floor(ijk / 2) and the coarse row of each fine voxel."""
    b, ijk = _unkey(keys)
    return torch.unique(_key(b, ijk >> 1), return_inverse=True)


def _rows2(keys, ckeys):
    """Fine rows under every coarse voxel for the 2^3 offsets, weight dimension 2 fastest."""
    b, ijk = _unkey(ckeys)
    return [_lookup(keys, b, 2 * ijk + torch.tensor([i, j, k], device=DEV, dtype=torch.int32))
            for i in (0, 1) for j in (0, 1) for k in (0, 1)]


def _wkio(w):
    """(Cout, Cin, K0, K1, K2) -> [K, Cin, Cout], K0 fastest."""
    return w.permute(4, 3, 2, 1, 0).reshape(-1, w.shape[1], w.shape[0])


def exact(case, seed):
    kind = case["kind"]
    if kind == "points":
        return None  # whole numbers
    w = {k: v.double() for k, v in _weights(case, seed).items()}
    keys, n_grids = _voxel_keys(case, seed)
    n = keys.numel()
    dt = _dtype(case)

    def feats(salt, rows, c):
        return _randn(seed, salt, (rows, c), dt).double()

    if kind == "groupnorm":
        b, _ = _unkey(keys)
        x = (_randn(seed, 2, (n, case["cin"]), torch.float32) * 1.5 + 0.5).to(dt).double().requires_grad_(True)
        gamma, beta = w["gamma"].requires_grad_(True), w["beta"].requires_grad_(True)
        parts = x.split(torch.bincount(b, minlength=n_grids).tolist())
        y = torch.cat([torch.nn.functional.group_norm(p.t()[None], case["groups"], gamma, beta)[0].t() for p in parts])
        g = torch.autograd.grad(y, [x, gamma, beta], feats(4, n, case["cin"]))
        return {"y": y.detach(), "dx": g[0], "dgamma": g[1], "dbeta": g[2]}
    if kind == "pool":
        x, dy = feats(2, n, case["cin"]), feats(4, n, case["cin"])
        ckeys, parent = _coarse(keys)
        idx = parent[:, None].expand_as(x)
        low = torch.zeros(ckeys.numel(), case["cin"], dtype=torch.float64, device=DEV)
        dlow = torch.zeros_like(low).index_add_(0, parent, dy)
        if case["mode"] == "max":
            low = low.scatter_reduce(0, idx, x, "amax", include_self=False)
            first = torch.full(low.shape, n, device=DEV)  # a window's gradient goes to its first maximum
            at = torch.where(x == low[parent], torch.arange(n, device=DEV)[:, None], n)
            first = first.scatter_reduce(0, idx, at, "amin")
            dx = torch.where(first[parent] == torch.arange(n, device=DEV)[:, None], dlow[parent], 0.0)
        else:
            low.index_add_(0, parent, x)
            low /= 8
            dx = dlow[parent] / 8
        return {"low": low, "up": low[parent], "dx": dx}
    if kind == "up":
        ckeys, parent = _coarse(keys)
        _, ijk = _unkey(keys)
        o = (ijk & 1).long()
        child = o[:, 0] * 4 + o[:, 1] * 2 + o[:, 2]
        x = feats(2, ckeys.numel(), case["cin"])
        wk = w["w1"].permute(4, 3, 2, 0, 1).reshape(8, case["cin"], case["cout"])
        rows = [torch.where(child == k, parent, -1) for k in range(8)]
        return {"y": _Conv64.apply(x, wk, rows) + w["w1_bias"]}
    rows = _rows3(keys)
    x = feats(2, n, case["cin"])
    if kind == "layer":
        return {"y": _Conv64.apply(x, _wkio(w["w1"]), rows) + w["w1_bias"]}
    if kind == "infer":
        h = _Conv64.apply(x, _wkio(w["w1"]), rows) + w["w1_bias"]
        if case["norm"]:
            h = (h - w["mean"]) * torch.rsqrt(w["var"] + 1e-5) * w["gamma"] + w["beta"]
        ckeys, _ = _coarse(keys)
        return {"y": _Conv64.apply(torch.relu(h), _wkio(w["w2"]), _rows2(keys, ckeys)) + w["w2_bias"]}
    if kind == "serve":
        for i in range(3):
            x = _Conv64.apply(x, _wkio(w["w%d" % i]), rows)
            x = torch.relu(x) if i < 2 else x
        return {"y": x, "ijk": None}
    x.requires_grad_(True)
    dy = feats(4, n, case["cout"])
    if kind == "halo":
        wt = w["w1"].requires_grad_(True)
        y = _Conv64.apply(x, _wkio(wt), rows)
        g = torch.autograd.grad(y, [x, wt], dy)
        return {"y": y.detach(), "dx": g[0], "dw": g[1]}
    ps = [w[k].requires_grad_(True) for k in ("w1", "w1_bias", "w2", "w2_bias")]
    h = torch.relu(_Conv64.apply(x, _wkio(ps[0]), rows) + ps[1])
    y = _Conv64.apply(h, _wkio(ps[2]), rows) + ps[3]
    g = torch.autograd.grad(y, [x, *ps], dy)
    return {"y": y.detach(), "dx": g[0], "dw1": g[1], "db1": g[2], "dw2": g[3], "db2": g[4]}
