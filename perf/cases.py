"""The performance cases of the framework: what its users run through its public entry points.

Five kinds of call, each over the sizes, element types and options it is used with:

  pass    W-MSA then SW-MSA over one scene: the two window plans from raw voxel coordinates
          (`window.bucket_windows`) and the fused attention core over given q, k, v rows
          (`attention.window_attention_fused`).  The new plan belongs to the call: every scene has its own.
  module  `WindowAttentionSparse.forward`, the drop-in of upstream's module: bucketing, qkv Linear,
          attention core, projection, and the default check of the device-side error word; as
          inference, as a training step (gradients of the input and of every parameter), or as the
          operator-by-operator chain on the COO surface (`fused=False`).
  stage   `BasicLayer.forward` on `SparseVoxels`: a whole Swin stage from coordinates and features,
          as inference or as a training step.
  conv    the sparse convolutions around the stages on a new coordinate set: two submanifold
          convolutions that share a rulebook (a residual block), patch merging and patch expansion.

Scenes.  `room`: the surface-sparse synthetic room of `scenes.room_scene`.  `spread` sets how many of
its surface cells are occupied: 1.0 is a raw scan at full resolution (a median of 9-11 voxels in a 7^3
window), 1.7 is what the strided convolutions leave for the deeper stages (33-46, up to 170).  The voxel
size follows from the voxel count.  `uniform`: cells drawn uniformly from a cube.  `skewed`: a share of
the 9^3 blocks completely full (729 voxels), the others nearly empty."""
from __future__ import annotations

import math

import numpy as np
import torch

from sparseswin3d_b200 import scenes
from sparseswin3d_b200.attention import WindowAttentionSparse, plan_params, window_attention_fused
from sparseswin3d_b200.sparse_conv import PatchExpand, PatchMerging, SubMConv3d
from sparseswin3d_b200.stage import BasicLayer, SparseVoxels
from sparseswin3d_b200.voxels import WindowedVoxels
from sparseswin3d_b200.window import bucket_windows, resolve_geometry, window_keys

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # The deepest Swin stage: few voxels, wide rows.  The smallest call a network makes: launches and
        # host work are most of it.
        dict(name="module_c384_2k5_bf16", kind="module", mode="infer", scene="room", n=2500, spread=1.7, batch=1, heads=12,
             head_dim=32, window=7, shift=3, dtype="bf16"),
        # A single attention module on volume-sparse points: 20 000 distinct cells of a 128^3 grid.
        dict(name="module_uniform_20k_f32", kind="module", mode="infer", scene="uniform", n=20000, grid=128, batch=1, heads=3,
             head_dim=32, window=7, shift=0, dtype="f32"),
        # The headline: W-MSA + SW-MSA on one indoor scan of 150 000 voxels, C = 96, in both precisions.
        dict(name="pass_room150k_f32", kind="pass", scene="room", n=150000, spread=1.0, batch=1, heads=3, head_dim=32, window=7,
             shift=3, dtype="f32"),
        dict(name="pass_room150k_bf16", kind="pass", scene="room", n=150000, spread=1.0, batch=1, heads=3, head_dim=32, window=7,
             shift=3, dtype="bf16"),
        # The largest: a million voxels, half of the 9^3 windows completely full, C = 192.
        dict(name="pass_skewed_1m_bf16", kind="pass", scene="skewed", grid=126, p_dense=0.5, batch=1, heads=6, head_dim=32,
             window=9, shift=0, dtype="bf16"),
        # A ragged batch in half precision with 16-channel heads: the first stage of a narrow network.
        dict(name="pass_batch4_33333_f16", kind="pass", scene="room", n=33333, spread=1.3, batch=4, heads=6, head_dim=16, window=7,
             shift=3, dtype="f16"),
        # The stages of a network in inference: the first one at full size in bf16, a deep one in fp32.
        dict(name="stage_room150k_bf16", kind="stage", mode="infer", depth=2, scene="room", n=150000, spread=1.0, batch=1, heads=3,
             head_dim=32, window=7, dtype="bf16"),
        dict(name="stage_c192_10k_f32", kind="stage", mode="infer", depth=6, scene="room", n=10000, spread=1.7, batch=1, heads=6,
             head_dim=32, window=7, dtype="f32"),
        # Training: the attention module on the full scan in fp32, a stage at the second resolution in bf16.
        dict(name="train_module_room150k_f32", kind="module", mode="train", scene="room", n=150000, spread=1.0, batch=1, heads=3,
             head_dim=32, window=7, shift=3, dtype="f32"),
        dict(name="train_stage_40k_bf16", kind="stage", mode="train", depth=2, scene="room", n=40000, spread=1.7, batch=1, heads=3,
             head_dim=32, window=7, dtype="bf16"),
        # A residual block, patch merging and patch expansion on a new scan.
        dict(name="conv_room150k_bf16", kind="conv", scene="room", n=150000, spread=1.0, batch=1, channels=48, dtype="bf16"),
        # Code written against upstream's operators: the unfused chain on a quarter of a scan.
        dict(name="ops_room36k_f32", kind="module", mode="ops", scene="room", n=35935, spread=1.0, batch=1, heads=3, head_dim=32,
             window=7, shift=3, dtype="f32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pass", "pass", "pass", "module", "module", "stage", "stage", "conv"])
    spread = rng.choice([1.0, 1.3, 1.7])
    if kind == "pass":
        if rng.random() < 0.3:
            dtype = rng.choice(["bf16", "f16", "f32"])
            grid = 9 * rng.randint(3, 7 if dtype == "f32" else 13)
            return dict(kind=kind, scene="skewed", grid=grid, p_dense=round(rng.uniform(0.2, 0.5), 2), batch=1,
                        heads=rng.choice([3, 6]), head_dim=32, window=9, shift=rng.choice([0, 4]), dtype=dtype)
        heads, head_dim = rng.choice([(3, 32), (6, 32), (3, 16), (6, 16), (12, 16)])
        return dict(kind=kind, scene="room", n=_log_int(rng, 2000, 150000), spread=spread, batch=rng.choice([1, 1, 2, 4]),
                    heads=heads, head_dim=head_dim, window=rng.choice([5, 7, 7]), shift=rng.choice([2, 2, 1]),
                    dtype=rng.choice(["f32", "bf16", "f16"]))
    if kind == "module":
        mode = rng.choice(["infer", "infer", "train", "ops"])
        top = {"infer": 150000, "train": 150000, "ops": 36000}[mode]
        heads, head_dim = rng.choice([(3, 32), (6, 32), (3, 16)])
        return dict(kind=kind, mode=mode, scene="room", n=_log_int(rng, 1000, top), spread=1.0 if mode == "ops" else spread,
                    batch=1, heads=heads, head_dim=head_dim, window=7, shift=rng.choice([0, 3]),
                    dtype="f32" if mode == "ops" else rng.choice(["f32", "bf16"]))
    if kind == "stage":
        heads, head_dim, top = rng.choice([(3, 16, 150000), (3, 32, 150000), (6, 32, 40000), (12, 32, 10000)])
        mode = rng.choice(["infer", "infer", "train"])
        dtype = rng.choice(["f32", "bf16"])
        if mode == "train" or dtype == "f32":
            top = min(top, 60000)
        return dict(kind=kind, mode=mode, depth=rng.choice([1, 2]), scene="room", n=_log_int(rng, 1500, top), spread=spread,
                    batch=rng.choice([1, 2]), heads=heads, head_dim=head_dim, window=7, dtype=dtype)
    return dict(kind=kind, scene="room", n=_log_int(rng, 3000, 150000), spread=spread, batch=rng.choice([1, 2]),
                channels=rng.choice([32, 48, 96]), dtype=rng.choice(["f32", "bf16", "f16"]))


# ---- inputs ------------------------------------------------------------------------------------
def _coords(case, seed):
    if case["scene"] == "uniform":
        c, dims = scenes.uniform_scene(case["n"], case["grid"], seed)
    elif case["scene"] == "skewed":
        c, dims = _skewed(case, seed)
    else:
        batch = case["batch"]
        share = [case["n"] // batch + (1 if b < case["n"] % batch else 0) for b in range(batch)]
        voxel = 0.02 * math.sqrt(150000 * batch / case["n"]) * case["spread"]
        parts = [scenes.room_scene(m, seed=seed * 16 + b, batch_index=b, voxel_m=voxel) for b, m in enumerate(share)]
        c, dims = np.concatenate([p[0] for p in parts]), parts[0][1]
    return torch.from_numpy(np.ascontiguousarray(c)).cuda(), dims


def _skewed(case, seed):
    """The blocks of `scenes.skewed_scene`, in numbers that do not depend on the seed: so many full, the
    others with 1-8 voxels in turn."""
    rng = np.random.default_rng(seed)
    nw, n = case["grid"] // 9, 729
    order = rng.permutation(nw ** 3)
    full = int(round(case["p_dense"] * nw ** 3))
    count = np.empty(nw ** 3, dtype=np.int64)
    count[order] = np.where(np.arange(nw ** 3) < full, n, np.arange(nw ** 3) % 8 + 1)
    w, p = np.nonzero(rng.permuted(np.tile(np.arange(n, dtype=np.int16), (nw ** 3, 1)), axis=1) < count[:, None])
    zyx = [(w // d % nw) * 9 + (p // e % 9) for d, e in ((nw * nw, 81), (nw, 9), (1, 1))]
    c = np.stack([np.zeros_like(w), *zyx], 1).astype(np.int32)
    return c[rng.permutation(len(c))], (case["grid"],) * 3


def _moved(case, seed):
    """One scan per size, moved about a slightly larger grid by whole 2-cells and listed in another order for
    every seed: the number of merged voxels is the same for all of them."""
    c, dims = _coords(case, case["n"])
    rng = np.random.default_rng(seed)
    step = torch.tensor([0, *(2 * rng.integers(0, 6, 3))], dtype=torch.int32, device="cuda")
    if seed % 2:
        c = c[:, [0, 2, 1, 3]]  # the room is as long as it is wide
    order = torch.from_numpy(rng.permutation(len(c))).cuda()
    return (c + step)[order].contiguous(), tuple((d + 11) // 2 * 2 for d in dims)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1 + seed)


def _table_rows(w):
    return (2 * w - 1) ** 3


def _fill(module, g):
    """Weights as a trained network has them: Linears at their fan-in's scale, norms near one, a bias
    table of moderate size."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            noise = torch.randn(p.shape, device=p.device, generator=g)
            if "relative_position_bias_table" in name:
                p.copy_(noise * 0.2)
            elif "norm" in name:
                p.copy_(1.0 + 0.1 * noise if name.endswith("weight") else 0.1 * noise)
            elif name.endswith("bias"):
                p.copy_(0.02 * noise)
            elif p.dim() == 3:  # convolution [k^3, Cin, Cout]
                p.copy_(noise / math.sqrt(p.shape[0] * p.shape[1]))
            else:
                p.copy_(noise / math.sqrt(p.shape[-1]))
    return module


def _mask(coords, geom):
    """(window, pos) of every voxel and, for a shifted geometry, the [windows, positions] mask table."""
    idx, region, _ = window_keys(coords, geom, with_region=True)
    if not geom.shifted:
        return idx, None
    mask = torch.zeros(geom.n_windows, geom.n_per_window, dtype=torch.int8, device="cuda")
    mask[idx[:, 0].long(), idx[:, 1].long()] = region
    return idx, mask


def prepare(case, seed):
    dtype = DTYPES[case["dtype"]]
    g = _generator(seed)
    coords, dims = (_moved if case["kind"] == "conv" else _coords)(case, seed)
    n = coords.shape[0]
    s = {"kind": case["kind"], "mode": case.get("mode", "infer"), "coords": coords}
    if case["kind"] == "conv":
        c = case["channels"]
        s["feats"] = torch.randn(n, c, device="cuda", generator=g).to(dtype)
        s["dims"], s["batch"] = dims, case["batch"]
        layers = torch.nn.ModuleList([SubMConv3d(c, c, 3, bias=False, indice_key="res"), SubMConv3d(c, c, 3, bias=False, indice_key="res"),
                                      PatchMerging(c, indice_key="down"), PatchExpand(2 * c, indice_key="down")])
        s["layers"] = _fill(layers.cuda(), g).to(dtype).eval()
        return s
    H, hd, w = case["heads"], case["head_dim"], (case["window"],) * 3
    C = H * hd
    if case["kind"] == "pass":
        shifts = [(0, 0, 0), (case["shift"],) * 3] if case["shift"] else [(0, 0, 0)]
        s["geoms"] = [resolve_geometry(case["batch"], dims, w, sh) for sh in shifts]
        s["params"] = plan_params(H, hd, dtype, w)
        s["qkv"] = [torch.randn(n, 3, H, hd, device="cuda", generator=g).to(dtype) for _ in shifts]
        s["table"] = torch.randn(_table_rows(case["window"]), H, device="cuda", generator=g) * 0.2
        s["scale"] = hd ** -0.5
        return s
    feats = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    if case["kind"] == "module":
        m = _fill(WindowAttentionSparse(C, H, w, qkv_bias=True).cuda(), g).to(dtype)
        geom = resolve_geometry(case["batch"], dims, w, (case["shift"],) * 3)
        idx, s["mask"] = _mask(coords, geom)
        s["x"] = WindowedVoxels(feats, idx, geom.n_windows, (geom.n_per_window,))
    else:
        m = _fill(BasicLayer(dim=C, depth=case["depth"], num_heads=H, window_size=w, qkv_bias=True).cuda(), g).to(dtype)
        s["x"] = SparseVoxels(feats, coords, dims, case["batch"])
    s["module"] = m
    if s["mode"] == "train":
        feats.requires_grad_(True)
        s["grad"] = torch.randn(n, C, device="cuda", generator=g).to(dtype)
    else:
        m.eval()
    return s


# ---- one pass ----------------------------------------------------------------------------------
def run(s):
    kind, mode = s["kind"], s["mode"]
    if kind == "pass":
        outs = []
        for geom, qkv in zip(s["geoms"], s["qkv"]):
            plan = bucket_windows(coords=s["coords"], geom=geom, **s["params"])
            outs.append(window_attention_fused(qkv, plan, s["table"], s["scale"], use_mask=bool(geom.shifted)))
        return outs
    if kind == "conv":
        with torch.no_grad():
            a, b, merge, expand = s["layers"]
            x = SparseVoxels(s["feats"], s["coords"], s["dims"], s["batch"])
            y = b(a(x))
            down = merge(y)
            up = expand(down)
        return [y.features, down.indices, down.features, up.features]
    m = s["module"]
    args = (s["x"], s["mask"]) if kind == "module" else (s["x"],)
    if mode == "train":
        params = [p for p in m.parameters()]
        y = m(*args).features
        return [y, *torch.autograd.grad(y, [s["x"].features, *params], s["grad"])]
    with torch.no_grad():
        return m(*args, fused=False).features if mode == "ops" else m(*args).features


# ---- what a pass cannot do without ---------------------------------------------------------------
def _size(case):
    """(voxels, sum over windows of c^2) of a scene, the latter as the generators give it on average."""
    if case["scene"] == "skewed":
        w = (case["grid"] // 9) ** 3
        full = int(round(case["p_dense"] * w))
        return full * 729 + int((w - full) * 4.5), full * 729 ** 2
    n = case["n"]
    if case["scene"] == "uniform":
        return n, n * (1 + n * case["window"] ** 3 / case["grid"] ** 3)
    return n, n * 12.5 * case["spread"] ** 2.6 * (case.get("window", 7) / 7) ** 2.2


def work(case):
    elt = 4 if case["dtype"] == "f32" else 2
    n, sq = _size(case)
    if case["kind"] == "conv":
        c = case["channels"]
        m, pairs = n * 0.55, n * 2.6 * case["spread"] ** 2   # merged voxels; (input, output) pairs of a 3^3 kernel
        flops = 2 * 2 * pairs * c * c + 2 * 2 * n * c * 2 * c
        return {"bytes": (n * c * 3 + m * 2 * c) * elt + n * 16 + m * 16, "flops": flops}
    C = case["heads"] * case["head_dim"]
    core = 4 * C * sq
    if case["kind"] == "pass":
        k = 2 if case["shift"] else 1
        return {"bytes": k * 4 * n * C * elt + n * 16 + _table_rows(case["window"]) * case["heads"] * 4, "flops": k * core}
    train = case["mode"] == "train"
    weights = 4 * C * C + 4 * C + _table_rows(case["window"]) * case["heads"]
    flops = 8 * n * C * C + core
    if case["kind"] == "stage":
        weights = (weights + 8 * C * C + 9 * C) * case["depth"]
        flops = (flops + 16 * n * C * C) * case["depth"]
    rows = 4 if train else 2                    # features in, result out; and both gradients
    return {"bytes": (rows * n * C + weights * (2 if train else 1)) * elt + n * 16, "flops": flops * (3 if train else 1)}


def tolerance(case):
    """Four times what each kind of path showed against itself: 16-bit cases against the same path in fp32 on
    the same rounded inputs and weights (attention core: bf16 1.7e-3, f16 2.5e-4, one rounding of the output;
    a module or layer chain: bf16 3.6e-3 to 4.9e-3, with gradients 7.7e-3, f16 convolutions 5.8e-4), fp32 cases
    against inputs moved by half a unit in the last place (up to 8e-7)."""
    if case["dtype"] == "f32":
        return {"rel": 4e-6, "max": 5e-5}
    half = 0.15 if case["dtype"] == "f16" else 1.0
    if case["kind"] == "pass":
        return {"rel": 6.6e-3 * half, "max": 1.6e-2 if case["dtype"] == "bf16" else 6.4e-3}
    if case.get("mode") == "train":
        return {"rel": 3e-2 * half, "max": 0.36 * half}
    return {"rel": 2e-2 * half, "max": 0.12 * half}
