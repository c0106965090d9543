"""The calls a user of this framework makes, over the sizes and options they are made with.

Three kinds of call reach the kernels when a Swin3D network runs:

* ``attn``     one window attention of a backbone block (``SelfAttnAIOFunction``), forward or forward
               and backward, in the three precision modes of ``WindowAttention(fp16_mode=0/1/2)``;
* ``windows``  the grouping of a stage's voxels into windows (``get_index01``), twice per stage;
* ``knn``      the neighbour search between two stages (``KNN``) and its two callers, the K = 3
               interpolation of ``Upsample`` and the K = 16 pooling of ``GridKNNDownsample``.

Inputs are synthetic indoor rooms (surface-sampled floor, ceiling, walls, boxes), seen by stage s on a
grid 2^(s-1) times coarser than the voxels, and point sets on random planes for the plain search.
The two backbones are Swin3D-S and Swin3D-L, quant_size 4.
"""
from types import SimpleNamespace

import numpy as np
import torch

from swin3d_b200 import synthetic as syn
from swin3d_b200.sparse_dl.attn.attn_coff import (IndexMode, PosEmb, PrecisionMode, SelfAttnAIOFunction,
                                                  TableDims)
from swin3d_b200.sparse_dl.knn import KNN, knn_linear_interpolation, knn_max_pool
from swin3d_b200.window import build_windows, get_index01

QUANT = 4
WINDOWS = (5, 7, 7, 7, 7)                                   # per stage
CHANNELS = {"S": (48, 96, 192, 384, 384), "L": (80, 160, 320, 640, 640)}
HEADS = {"S": (6, 6, 12, 24, 24), "L": (10, 10, 20, 40, 40)}
SIGNALS = {"XYZ": 3, "XYZ_RGB": 6, "XYZ_RGB_NORM": 9}
# fp16_mode of WindowAttention: 0 everything fp32, 1 fp16 forward and fp32 backward, 2 everything fp16
PRECISION = {0: PrecisionMode.HALF_NONE, 1: PrecisionMode.HALF_FORWARD, 2: PrecisionMode.HALF_ALL}


def _attn(name, model, stage, rooms, voxels, fp16_mode, train, crse="XYZ_RGB_NORM", shift=False):
    return {"name": name, "kind": "attn", "model": model, "stage": stage, "rooms": rooms, "voxels": voxels,
            "fp16_mode": fp16_mode, "train": train, "crse": crse, "shift": shift}


def _windows(name, stage, rooms, voxels, shift, crse="XYZ_RGB_NORM"):
    return {"name": name, "kind": "windows", "stage": stage, "rooms": rooms, "voxels": voxels, "shift": shift,
            "crse": crse}


def _knn(name, op, points, scenes, n_src, n_query, channels, half, train):
    return {"name": name, "kind": "knn", "op": op, "points": points, "scenes": scenes, "n_src": n_src,
            "n_query": n_query, "channels": channels, "half": half, "train": train}


def listed():
    return [
        # training: first stage of Swin3D-L on a batch of eight rooms (964 k voxels, about 29 voxels per window)
        _attn("attn-L1-train-8rooms", "L", 1, 8, 125_000, 2, True),
        # training: second stage, head_dim 16 and windows of 7^3 cells, the shape of all later stages
        _attn("attn-L2-train-4rooms", "L", 2, 4, 150_000, 2, True, shift=True),
        # training: a late stage, many heads over a few thousand voxels
        _attn("attn-L4-train-4rooms", "L", 4, 4, 150_000, 2, True),
        # inference of one room: Swin3D-S, fp16_mode=1, forward only
        _attn("attn-S1-infer-room", "S", 1, 1, 120_000, 1, False),
        # the default mixed mode in training: fp16 forward, fp32 backward
        _attn("attn-S1-train-mixed", "S", 1, 1, 120_000, 1, True, shift=True),
        # a single small fp32 layer (colour signals only), as in a unit-sized model or a gradient check
        _attn("attn-layer-fp32", "S", 1, 1, 4_096, 0, True, crse="XYZ_RGB"),
        # inference, deepest stage of one room: a few hundred voxels, launches and host work
        _attn("attn-S5-infer-room", "S", 5, 1, 120_000, 2, False),
        # window grouping of the training batch, shifted windows
        _windows("windows-8rooms", 1, 8, 125_000, True),
        # window grouping of a deep stage of one room
        _windows("windows-room-stage4", 4, 1, 120_000, False),
        # decoder: features of 50 k coarse points interpolated at 200 k fine points in each of eight scenes
        _knn("knn-upsample-8scenes", "upsample", "planes", 8, 50_000, 200_000, 80, True, True),
        # encoder: stage 1 to stage 2 of four rooms, 16 neighbours pooled
        _knn("knn-downsample-4rooms", "downsample", "rooms", 4, 120_000, 30_000, 160, True, True),
        # the plain search between two deep stages of one room
        _knn("knn-search-room", "search16", "rooms", 1, 2_000, 500, 0, False, False),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["attn"] * 5 + ["windows"] * 2 + ["knn"] * 3)
    crse = rng.choice(["XYZ_RGB_NORM", "XYZ_RGB_NORM", "XYZ_RGB"])
    if kind == "attn":
        c = _attn("", rng.choice("SL"), rng.randint(1, 5), rng.randint(1, 8), _log_int(rng, 4_000, 150_000),
                  rng.choice([0, 1, 2, 2]), rng.random() < 0.6, crse, rng.random() < 0.5)
        # no dearer than the first listed case: a pair costs several times more in fp32
        while _pairs(c) * HEADS[c["model"]][c["stage"] - 1] * (1 if c["fp16_mode"] == 2 else 6) > 2.2e8:
            c["rooms"], c["voxels"] = max(1, c["rooms"] - 1), int(c["voxels"] * 0.9)
    elif kind == "windows":
        c = _windows("", rng.randint(1, 5), rng.randint(1, 8), _log_int(rng, 4_000, 150_000), rng.random() < 0.5, crse)
    else:
        op = rng.choice(["upsample", "downsample", "search3", "search16"])
        scenes = rng.randint(1, 8)
        up = op in ("upsample", "search3")
        coarse = _log_int(rng, 400, 50_000)
        fine = int(coarse * rng.uniform(3.0, 4.5))
        if not up:
            fine = min(fine, 150_000)
        # no dearer than the listed searches, counted in pairs of points of a scene
        while scenes > 1 and scenes * coarse * fine > (4e10 if up else 1.4e10):
            scenes -= 1
        if scenes > 1:                                       # sources of several scenes begin at multiples of four
            coarse, fine = (coarse // 4 * 4, fine) if up else (coarse, fine // 4 * 4)
        c = _knn("", op, rng.choice(["planes", "rooms"]), scenes, coarse if up else fine, fine if up else coarse,
                 0 if op.startswith("search") else rng.choice([48, 80, 96, 160, 320]), rng.random() < 0.6,
                 not op.startswith("search") and rng.random() < 0.6)
    del c["name"]
    return c


# ---- sizes ------------------------------------------------------------------------------------------

def _voxels(case):
    """Voxels of the case: a surface loses three quarters of its voxels from one stage to the next."""
    return case["rooms"] * case["voxels"] * 0.96 / 4 ** (case["stage"] - 1)


def _pairs(case):
    """Attention pairs: a window holds a piece of surface, about ws^2 voxels, somewhat more at corners."""
    return _voxels(case) * min(1.15 * WINDOWS[case["stage"] - 1] ** 2, max(1.0, _voxels(case)))


def work(case):
    if case["kind"] == "attn":
        s = case["stage"] - 1
        n, C, H, D = _voxels(case), CHANNELS[case["model"]][s], HEADS[case["model"]][s], SIGNALS[case["crse"]]
        b = 4 if case["fp16_mode"] == 0 else 2
        table = sum(_sizes(case))
        # q, k, v read and out written; coordinates and the row list; the tables
        nbytes = n * (4 * C * b + 4 * D + 4) + 3 * table * 4
        flops = 4.0 * _pairs(case) * C + 3.0 * D * _pairs(case) * H
        if case["train"]:                                    # q, k, v, out, dout read; dq, dk, dv written
            nbytes += n * (8 * C * b + 4 * D + 4 + 4 * H) + 6 * table * 4
            flops += 10.0 * _pairs(case) * C + 6.0 * D * _pairs(case) * H
        return {"bytes": nbytes, "flops": flops}
    if case["kind"] == "windows":
        # coordinates and signals read; order, signals in the new order and the window lists written
        n, D = _voxels(case), SIGNALS[case["crse"]]
        return {"bytes": n * (16 + 4 * D + 4 + 4 * D + 24 / 20), "flops": 0}
    nq, ns, C = case["scenes"] * case["n_query"], case["scenes"] * case["n_src"], case["channels"]
    K, b = _k(case), 2 if case["half"] else 4
    nbytes = 12.0 * (nq + ns)
    if case["op"].startswith("search"):
        nbytes += 8.0 * K * nq
    else:
        nbytes += (nq + ns) * C * b * (2 if case["train"] else 1)
    # a search structure visits some tens of points per query for a handful of neighbours
    return {"bytes": nbytes, "flops": nq * (8.0 * 4 * K + 2.0 * K * C * (2 if case["train"] else 1))}


def tolerance(case):
    if case["kind"] == "attn":
        # fp32 sums; fp16 storage with fp32 accumulation, table gradients summed over all windows
        return {"rel": 1e-5, "max": 1e-3} if case["fp16_mode"] == 0 else {"rel": 5e-3, "max": 0.2}
    if case["kind"] == "windows" or case["op"].startswith("search"):
        return "exact"
    return {"rel": 1e-3, "max": 2e-2} if case["half"] else {"rel": 1e-5, "max": 1e-3}


# ---- inputs -----------------------------------------------------------------------------------------

def _k(case):
    return 3 if case["op"] in ("upsample", "search3") else 16


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _stage(case, seed):
    """Voxel coordinates (batch, x, y, z) int32 and signals (in-voxel position, colour, normal) of the
    case's rooms as its stage sees them.  The shape of the rooms belongs to the case, so that every
    seed has as many voxels and windows; where the rooms stand (by whole windows), at which voxel
    the list begins and all signals but the normals come from the seed."""
    s = case["stage"] - 1
    sc = syn.concat_scenes([syn.make_room(case["rooms"] * 8 + r, case["voxels"]) for r in range(case["rooms"])])
    coords, feats = _coarser(torch.from_numpy(sc.coords).cuda(),
                             torch.from_numpy(syn.signal_feats(sc, case["crse"])).cuda(), 1 << s)
    g, rng, n = _gen(seed), np.random.default_rng(seed), coords.shape[0]
    first = int(rng.integers(n))
    coords, feats = coords.roll(first, 0), feats.roll(first, 0)
    step = torch.from_numpy(rng.integers(0, 16, 3).astype(np.int32)).cuda()
    coords[:, 1:] += step * (WINDOWS[s] << s)
    feats[:, :min(6, feats.shape[1])] = torch.rand((n, min(6, feats.shape[1])), generator=g, device="cuda")
    return coords.contiguous(), feats.contiguous()


def _coarser(coords, feats, stride):
    """What a stage `stride` times coarser sees: the first voxel of every coarse cell stands for it."""
    if stride == 1:
        return coords, feats
    c = coords.clone()
    c[:, 1:] = torch.div(c[:, 1:], stride, rounding_mode="floor") * stride
    x = c.long()
    key = ((x[:, 0] << 48) | (x[:, 1] << 32) | (x[:, 2] << 16) | x[:, 3])
    _, inverse = torch.unique(key, return_inverse=True)
    first = torch.full((int(inverse.max()) + 1,), c.shape[0], dtype=torch.int64, device=c.device)
    first.scatter_reduce_(0, inverse, torch.arange(c.shape[0], device=c.device), "amin")
    first = first.sort().values
    return c[first].contiguous(), feats[first].contiguous()


def _sizes(case):
    s = case["stage"] - 1
    H = HEADS[case["model"]][s]
    return syn.table_sizes(WINDOWS[s], QUANT, H, CHANNELS[case["model"]][s] // H, case["crse"])


def _shift(case):
    return WINDOWS[case["stage"] - 1] // 2 if case["shift"] else 0


def _prepare_attn(case, seed):
    s = case["stage"] - 1
    H, hd = HEADS[case["model"]][s], CHANNELS[case["model"]][s] // HEADS[case["model"]][s]
    coords, feats = _stage(case, seed)
    wi = build_windows(coords, feats, WINDOWS[s], _shift(case), 1 << s)
    crse = wi.n_coords.clone()                               # the signals in table units
    crse[:, :3] *= QUANT
    crse[:, 3:] *= 2 * QUANT
    g, n, sizes = _gen(seed), coords.shape[0], _sizes(case)
    # the qkv projection runs under autocast in the fp16 modes; the tables are fp32 parameters
    act = torch.float32 if case["fp16_mode"] == 0 else torch.float16
    q, k, v, grad = (torch.randn((n, H, hd), generator=g, device="cuda").to(act) for _ in range(4))
    q *= hd ** -0.5
    tables = [torch.nn.init.trunc_normal_(torch.empty(sum(sizes), device="cuda"), std=0.02, a=-0.04, b=0.04,
                                          generator=g) for _ in range(3)]
    leaves = [q, k, v, *tables]
    for t in leaves:
        t.requires_grad_(case["train"])
    return SimpleNamespace(kind="attn", leaves=leaves, grad=grad, indices=wi.reference_indices(crse), train=case["train"],
                           offsets=torch.tensor(sizes, dtype=torch.int32, device="cuda"),
                           autocast=case["fp16_mode"] != 0, precision=PRECISION[case["fp16_mode"]])


def _prepare_windows(case, seed):
    coords, feats = _stage(case, seed)
    sp = SimpleNamespace(C=coords, tensor_stride=1 << (case["stage"] - 1))
    return SimpleNamespace(kind="windows", sp=sp, local=feats[:, :3].contiguous(), colors=feats[:, 3:].contiguous(),
                           window=WINDOWS[case["stage"] - 1], shift=_shift(case))


def _room_points(seed, fine, coarse):
    """Positions of a room's voxels and the subset of them that stands for the next stage."""
    rng = np.random.default_rng(seed)
    room = syn.make_room(seed, max(int(fine * 1.5), 4_000))
    p = (room.coords[:, 1:] + room.local).astype(np.float32)
    p = p[np.sort(rng.choice(p.shape[0], size=min(fine, p.shape[0]), replace=False))]
    return p, p[np.sort(rng.choice(p.shape[0], size=min(coarse, p.shape[0]), replace=False))]


def _prepare_knn(case, seed):
    up = case["n_query"] >= case["n_src"]
    src, query = [], []
    for b in range(case["scenes"]):
        if case["points"] == "planes":
            s, q = syn.make_knn_scene(seed * 64 + b, case["n_query"], case["n_src"])
        else:
            f, c = _room_points(seed * 64 + b, max(case["n_src"], case["n_query"]), min(case["n_src"], case["n_query"]))
            s, q = (c, f) if up else (f, c)
        src.append(s)
        query.append(q)

    def cloud(parts):
        ends = np.cumsum([p.shape[0] for p in parts]).astype(np.int32)
        return torch.from_numpy(np.concatenate(parts)).cuda(), torch.from_numpy(ends).cuda()

    (xs, os_), (xq, oq) = cloud(src), cloud(query)
    g, dt = _gen(seed), torch.float16 if case["half"] else torch.float32
    feats = torch.randn((xs.shape[0], case["channels"]), generator=g, device="cuda").to(dt).requires_grad_(case["train"])
    grad = torch.randn((xq.shape[0], case["channels"]), generator=g, device="cuda").to(dt)
    return SimpleNamespace(kind="knn", op=case["op"], K=_k(case), src=xs, query=xq, so=os_, qo=oq, feats=feats, grad=grad,
                           train=case["train"])


def prepare(case, seed):
    return {"attn": _prepare_attn, "windows": _prepare_windows, "knn": _prepare_knn}[case["kind"]](case, seed)


# ---- one pass ---------------------------------------------------------------------------------------

def _run_attn(s):
    with torch.set_grad_enabled(s.train), torch.autocast("cuda", dtype=torch.float16, enabled=s.autocast):
        out = SelfAttnAIOFunction.apply(*s.leaves, s.offsets, s.indices, PosEmb.SEPARATE, TableDims.D0,
                                        IndexMode.INDIRECT, s.precision)
    return (out, *torch.autograd.grad(out, s.leaves, s.grad)) if s.train else out


def _run_knn(s):
    with torch.set_grad_enabled(s.train):
        if s.op.startswith("search"):
            return KNN.apply(s.K, s.src, s.query, s.so, s.qo)
        if s.op == "upsample":
            out = knn_linear_interpolation(s.src, s.query, s.feats, s.so, s.qo, s.K)
        else:
            out = knn_max_pool(s.K, s.src, s.query, s.feats, s.so, s.qo)
    return (out, *torch.autograd.grad(out, [s.feats], s.grad)) if s.train else out


def run(state):
    if state.kind == "attn":
        return _run_attn(state)
    if state.kind == "windows":
        return get_index01(state.sp, state.local, state.colors, state.window, state.shift)
    return _run_knn(state)
