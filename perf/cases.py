"""Performance cases: the work that programs built on the ``ash`` package have it do.

Seven kinds of work, each through the public Python API:

  hash     fill an emptied map, look a batch up, erase a quarter of the keys, look the batch up again
  query    interpolate a batch of positions and backpropagate, with each gradient mode of the grid
  eikonal  the same with a loss on the spatial gradient (double backward)
  fuse     integrate RGB-D frames into a truncated-signed-distance volume
  mesh     marching cubes over such a volume
  smooth   Gaussian filter over the embeddings
  render   volume rendering of a batch of rays, as a training step or as an image

All inputs are synthetic and made from the seed.  Grids are given their blocks through the engine's
checkpoint format, so that a block has the same row in every process and whole tables can be compared.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("torch-ash_b200"))

import ash  # noqa: E402
from ash.fusion import TSDFFusion  # noqa: E402
from ash.render import SDFToDensity, render_rays  # noqa: E402

DEVICE = "cuda"


# ----------------------------------------------------------------------------------------- cases
def listed():
    return [
        # A few scans' worth of voxel keys with their values: the smallest useful map, launch-bound.
        {"name": "hash_100k", "kind": "hash", "keys": 100_000, "capacity": 200_000, "dim": 3, "valued": True,
         "duplicates": 0.0, "hits": 0.5, "clustered": False},
        # City-scale voxel set: far beyond the L2 cache, half of the inserted keys repeated.
        {"name": "hash_50m", "kind": "hash", "keys": 50_000_000, "capacity": 64_000_000, "dim": 3, "valued": False,
         "duplicates": 0.5, "hits": 0.5, "clustered": True},
        # Signed-distance field of an object: small table, small batch, one channel.
        {"name": "query_100k", "kind": "query", "points": 100_000, "blocks": 2_048, "grid_dim": 8, "channels": 1,
         "interpolation": "linear", "mode": "dense", "positions": True},
        # Feature grid of a large scene (a 16 GB table), a training batch of millions of points.
        {"name": "query_4m", "kind": "query", "points": 4_000_000, "blocks": 500_000, "grid_dim": 8, "channels": 16,
         "interpolation": "linear", "mode": "dense", "positions": True},
        # The same kind of field trained with sparse updates: only the touched rows are stepped.
        {"name": "rows_1m", "kind": "query", "points": 1_000_003, "blocks": 250_000, "grid_dim": 8, "channels": 16,
         "interpolation": "smooth_step", "mode": "row_list", "positions": False},
        # Signed distance and features trained with an eikonal term, at an odd batch size.
        {"name": "eikonal_700k", "kind": "eikonal", "points": 700_001, "blocks": 60_000, "grid_dim": 8, "channels": 8,
         "interpolation": "smooth_step", "mode": "dense"},
        # Live reconstruction: one camera frame into an existing volume.
        {"name": "frame_vga", "kind": "fuse", "frames": 1, "height": 480, "width": 640, "voxel": 0.015, "dilation": 1},
        # Offline reconstruction: a recording into an empty volume.
        {"name": "scan_vga", "kind": "fuse", "frames": 100, "height": 480, "width": 640, "voxel": 0.015, "dilation": 1},
        # Triangle mesh of a reconstructed room.
        {"name": "mesh_24k", "kind": "mesh", "blocks": 24_000, "grid_dim": 8},
        # Initialisation of a radiance field: 7x7x7 smoothing of signed distance and colour at resolution 512.
        {"name": "smooth_27k", "kind": "smooth", "blocks": 27_000, "capacity": 80_000, "grid_dim": 8, "channels": 4,
         "size": 7},
        # One training step of that field: 8192 rays of up to 128 samples.
        {"name": "render_8k", "kind": "render", "rays": 8_192, "samples": 128, "blocks": 27_000, "capacity": 80_000,
         "channels": 4, "interpolation": "linear", "train": True},
        # A whole 640 x 480 view of it.
        {"name": "view_300k", "kind": "render", "rays": 307_200, "samples": 128, "blocks": 27_000, "capacity": 80_000,
         "channels": 4, "interpolation": "linear", "train": False},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, uniform over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hash", "query", "query", "eikonal", "fuse", "mesh", "smooth", "render"])
    if kind == "hash":
        n = _spread(rng, 1_000, 30_000_000)
        return {"kind": kind, "keys": n, "capacity": int(n * rng.uniform(1.0, 2.0)), "dim": rng.choice([1, 2, 3, 3, 3, 4]),
                "valued": rng.random() < 0.5, "duplicates": rng.choice([0.0, 0.5]), "hits": round(rng.uniform(0.1, 1.0), 2),
                "clustered": rng.random() < 0.5}
    if kind in ("query", "eikonal"):
        channels, grid_dim = rng.choice([1, 2, 3, 4, 5, 8, 13, 16]), rng.choice([4, 8, 8, 8, 16])
        most = min(300_000, int(8e9 / (4 * channels * grid_dim**3)))
        case = {"kind": kind, "points": _spread(rng, 1_000, 3_000_000 if kind == "query" else 1_000_000),
                "blocks": _spread(rng, 200, most if kind == "query" else min(most, 80_000)), "grid_dim": grid_dim,
                "channels": channels, "interpolation": rng.choice(["linear", "smooth_step"]),
                "mode": rng.choice(["dense", "dense", "in_place", "row_list"])}
        if kind == "query":
            case["positions"] = rng.random() < 0.5
        elif case["mode"] == "row_list":
            case["mode"] = "dense"
        return case
    if kind == "fuse":
        height, width = rng.choice([(120, 160), (240, 320), (479, 637), (480, 640)])
        return {"kind": kind, "frames": _spread(rng, 1, 60), "height": height, "width": width,
                "voxel": round(rng.uniform(0.012, 0.03), 4), "dilation": rng.choice([1, 1, 2])}
    if kind == "mesh":
        grid_dim = rng.choice([4, 8, 8, 16])
        return {"kind": kind, "blocks": _spread(rng, 200, 24_000 if grid_dim <= 8 else 6_000), "grid_dim": grid_dim}
    if kind == "smooth":
        blocks = _spread(rng, 200, 27_000)
        return {"kind": kind, "blocks": blocks, "capacity": int(blocks * rng.uniform(1.0, 3.0)), "grid_dim": rng.choice([4, 8]),
                "channels": rng.choice([1, 2, 3, 4, 5, 8, 16]), "size": rng.choice([3, 5, 7])}
    train = rng.random() < 0.6
    blocks = _spread(rng, 2_000, 40_000)
    return {"kind": kind, "rays": _spread(rng, 100, 60_000 if train else 300_000), "samples": rng.choice([48, 64, 100, 128]),
            "blocks": blocks, "capacity": int(blocks * rng.uniform(1.0, 3.0)), "channels": rng.choice([4, 4, 5, 8]),
            "interpolation": rng.choice(["linear", "smooth_step"]), "train": train}


# ----------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _load_blocks(grid, coords):
    """Make ``coords`` (n, 3) the active blocks of ``grid``, block i in row i, as loading a checkpoint does."""
    engine, n = grid.engine, coords.shape[0]
    keys = torch.zeros((engine.capacity, 3), dtype=torch.int32, device=DEVICE)
    indices = torch.zeros(engine.capacity, dtype=torch.long, device=DEVICE)
    keys[:n], indices[:n] = coords, torch.arange(n, device=DEVICE)
    engine.load_state_dict({
        "_heap": torch.arange(engine.capacity, dtype=torch.int32, device=DEVICE), "_keys": keys, "_indices": indices,
        "_size": torch.tensor([n], dtype=torch.int32, device=DEVICE)})


def _ball_blocks(n, g, n_balls=64):
    """n distinct block coordinates in solid balls of about equal size: the interior of a scene, where
    nearly every block has all of its neighbours."""
    n_balls = max(1, min(n_balls, n // 100))
    each = -(-n // n_balls)
    reach = int(math.ceil((3.0 * each / (4.0 * math.pi)) ** (1 / 3))) + 2
    r = torch.arange(-reach, reach + 1, device=DEVICE, dtype=torch.int32)
    ball = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).view(-1, 3)
    ball = ball[torch.argsort(ball.float().norm(dim=1), stable=True)[:each]]
    side = int(math.ceil(n_balls ** (1 / 3)))
    places = torch.randperm(side**3, generator=g, device=DEVICE)[:n_balls]
    centres = torch.stack([places % side, (places // side) % side, places // side**2], 1).int() * (4 * reach)
    centres = centres + torch.randint(-reach, reach + 1, (n_balls, 3), generator=g, device=DEVICE, dtype=torch.int32)
    return (centres[:, None, :] + ball[None, :, :]).view(-1, 3)[:n].contiguous()


def _points_in(blocks, n, grid_dim, g):
    """n positions (cell units) uniform in randomly chosen blocks."""
    pick = torch.randint(blocks.shape[0], (n,), generator=g, device=DEVICE)
    return (blocks[pick].float() + torch.rand(n, 3, generator=g, device=DEVICE)) * grid_dim


def _room(g):
    """A room of 20 spheres in the cube [-1, 1]^3: (centres, radii)."""
    centres = (torch.rand(20, 3, generator=g, device=DEVICE) - 0.5) * 1.6
    return centres, 0.06 + 0.14 * torch.rand(20, generator=g, device=DEVICE)


def _room_distance(room, p):
    """Signed distance of positions p (..., 3) to the spheres and the walls at +-0.97."""
    d = 0.97 - p.abs().amax(-1)
    for c, r in zip(*room):
        d = torch.minimum(d, (p - c).norm(dim=-1) - r)
    return d


def _room_blocks(n, room, g):
    """The n blocks of a lattice over [-1, 1]^3 nearest to the room's surfaces: ((n, 3) coordinates from 0, lattice side)."""
    side = max(4, int(math.ceil(math.sqrt(n / 6.0))))
    r = torch.arange(side, device=DEVICE, dtype=torch.int32)
    lattice = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).view(-1, 3)
    near = _room_distance(room, (lattice.float() + 0.5) * (2.0 / side) - 1.0).abs()
    blocks = lattice[torch.argsort(near, stable=True)[:n]]
    return blocks[torch.randperm(blocks.shape[0], generator=g, device=DEVICE)].contiguous(), side


def _room_grid(case, g):
    """A bounded grid over the room whose blocks lie along its surfaces: (grid, room)."""
    room = _room(g)
    blocks, side = _room_blocks(case["blocks"], room, g)
    grid = ash.BoundedSparseDenseGrid(3, max(case["capacity"], blocks.shape[0]), case["channels"],
                                      grid_dim=case.get("grid_dim", 8), sparse_grid_dim=side, device=DEVICE)
    _load_blocks(grid, blocks)
    return grid, room


# ----------------------------------------------------------------------------------------- hash
def _prepare_hash(case, g):
    n, dim = case["keys"], case["dim"]
    span = {1: 2**30, 2: 2**15, 3: 2**18, 4: 2**18}[dim]

    def keys_of(m):
        if not case["clustered"]:
            return torch.randint(-span, span, (m, dim), generator=g, device=DEVICE, dtype=torch.int32)
        centres = torch.randint(-span, span, (1024, dim), generator=g, device=DEVICE).float()
        spread = {1: 2.0**20, 2: 2.0**10, 3: 512.0, 4: 512.0}[dim]
        which = torch.randint(1024, (m,), generator=g, device=DEVICE)
        return (centres[which] + spread * torch.randn(m, dim, generator=g, device=DEVICE)).round().to(torch.int32)

    fresh = keys_of(max(1, int(n * (1.0 - case["duplicates"]))))
    again = torch.randint(fresh.shape[0], (n - fresh.shape[0],), generator=g, device=DEVICE)
    keys = torch.cat([fresh, fresh[again]])[torch.randperm(n, generator=g, device=DEVICE)].contiguous()
    n_hit = int(n * case["hits"])
    queries = torch.cat([keys[torch.randint(n, (n_hit,), generator=g, device=DEVICE)], keys_of(n - n_hit)])
    queries = queries[torch.randperm(n, generator=g, device=DEVICE)].contiguous()
    state = {"keys": keys, "queries": queries, "erased": keys[: n // 4].contiguous()}
    if case["valued"]:
        state["map"] = ash.HashMap(dim, {"sdf": 1, "rgb": 3}, case["capacity"], DEVICE)
        # a repeated key repeats its value: which copy of a key wins an insertion is not defined
        f = keys.float().sum(dim=1, keepdim=True)
        state["values"] = {"sdf": torch.sin(f), "rgb": torch.cat([torch.cos(f), f * 1e-6, keys[:, :1].float()], dim=1).contiguous()}
    else:
        state["map"] = ash.HashSet(dim, case["capacity"], DEVICE)
    return state


def _run_hash(s):
    m = s["map"]
    m.clear()
    if "values" not in s:
        m.insert(s["keys"])
        before = m.find(s["queries"])
        m.erase(s["erased"])
        return before, m.find(s["queries"])
    m.insert(s["keys"], s["values"])
    before, values = m.find(s["queries"], return_indices=False, return_values=True)
    found = {name: torch.where(before.view(-1, 1), v, 0.0) for name, v in values.items()}  # a miss has no value
    m.erase(s["erased"])
    after, _ = m.find(s["queries"])
    return before, found, after


def _work_hash(case):
    n, dim, row = case["keys"], case["dim"], 16 if case["valued"] else 0
    slot = 32 if dim == 4 else 16
    new = n * (1.0 - case["duplicates"])
    insert = n * 4 * dim + new * (slot + 2 * row)
    find = n * (4 * dim + 1 + row) + n * case["hits"] * (slot + row)
    erase = n // 4 * 4 * dim + new / 4 * slot
    return {"bytes": insert + 2 * find - n * row + erase, "flops": 0}


# ----------------------------------------------------------------------------------------- query, eikonal
def _prepare_query(case, g):
    D, G = case["channels"], case["grid_dim"]
    blocks = _ball_blocks(case["blocks"], g)
    grid = ash.SparseDenseGrid(3, blocks.shape[0], D, G, DEVICE)
    _load_blocks(grid, blocks)
    grid.embeddings.data.normal_(0, 0.1, generator=g)
    grid.grad_mode = case["mode"]
    grid.construct_grid_neighbor_lut_(radius=1, bidirectional=False)
    x = _points_in(blocks, case["points"], G, g)
    z = torch.randn(case["points"], D, generator=g, device=DEVICE)
    return {"grid": grid, "x": x.requires_grad_(case.get("positions", True)), "z": z, "interpolation": case["interpolation"]}


def _clear_gradients(s):
    grid = s["grid"]
    s["x"].grad = None
    if grid.grad_mode == "in_place":
        grid.zero_grad_rows_(s["x"])
    else:
        grid.embeddings.grad = None


def _run_query(s):
    grid, x = s["grid"], s["x"]
    _clear_gradients(s)
    y, masks = grid(x, interpolation=s["interpolation"])
    y.backward(s["z"])
    if grid.grad_mode == "row_list":
        grid.apply_row_list_(alpha=-1e-3)
        grid.embeddings.grad = None
        return y, masks, x.grad, grid.embeddings.data
    return y, masks, x.grad, grid.embeddings.grad


def _run_eikonal(s):
    grid, x = s["grid"], s["x"]
    _clear_gradients(s)
    y, masks = grid(x, interpolation=s["interpolation"])
    (slope,) = torch.autograd.grad(y, x, s["z"], create_graph=True)
    loss = y.square().sum() + (slope.norm(dim=-1) - 1).square().sum()
    loss.backward()
    return y, masks, slope, x.grad, grid.embeddings.grad


def _work_query(case):
    n, D, G = case["points"], case["channels"], case["grid_dim"]
    table = case["blocks"] * G**3 * D * 4
    rows = table * -math.expm1(-n * 8 * D * 4 / table)    # the corner rows of the batch, each once where they overlap
    n_pos = n * 12
    forward = n_pos + rows + n * (4 * D + 1)
    eikonal = case["kind"] == "eikonal"
    positions = eikonal or case["positions"]
    backward = n * 4 * D + n_pos + (rows + n_pos if positions else 0)
    if case["mode"] == "row_list":
        backward += 2 * rows              # the touched rows of the parameters, read and written
    elif case["mode"] == "in_place":
        backward += 3 * rows              # cleared, then read and written
    else:
        backward += table                 # a whole gradient comes out
    if eikonal:
        backward += rows + n_pos + n * 4 * D   # the gradient of the slope, into the same table
    return {"bytes": forward + backward, "flops": n * 8 * D * (2 + 2 + (2 if positions else 0) + (4 if eikonal else 0))}


# ----------------------------------------------------------------------------------------- fuse
def _camera(eye, target):
    """Camera-to-world pose at ``eye`` looking at ``target``: +z forward, +x right, +y down."""
    forward = torch.nn.functional.normalize(target - eye, dim=0)
    right = torch.nn.functional.normalize(torch.linalg.cross(forward, torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64)), dim=0)
    pose = torch.eye(4, dtype=torch.float64)
    pose[:3, 0], pose[:3, 1], pose[:3, 2], pose[:3, 3] = right, torch.linalg.cross(forward, right), forward, eye
    return pose


def _room_frame(room, K, pose, height, width):
    """Depth (H, W) in metres and colour (H, W, 3) of a 10 m room of spheres seen from ``pose``."""
    centres, radii = room[0] * 5.0, room[1] * 5.0
    v, u = torch.meshgrid(torch.arange(height, device=DEVICE), torch.arange(width, device=DEVICE), indexing="ij")
    pose = pose.float().to(DEVICE)
    d = torch.stack([(u - K[0, 2]) / K[0, 0], (v - K[1, 2]) / K[1, 1], torch.ones_like(u, dtype=torch.float32)], -1)
    d, o = d.view(-1, 3) @ pose[:3, :3].T, pose[:3, 3]
    a, b = (d * d).sum(-1, keepdim=True), d @ (o - centres).T
    root = b * b - a * (((o - centres) ** 2).sum(-1) - radii**2)
    t = (-b - root.clamp_min(0).sqrt()) / a
    t_sphere, which = torch.where((root > 0) & (t > 1e-3), t, math.inf).min(dim=1)
    t_wall = torch.where(d > 0, (5.0 - o) / d, (-5.0 - o) / d).nan_to_num(math.inf).amin(dim=1)
    depth = torch.minimum(t_sphere, t_wall)
    color = 0.5 + 0.5 * torch.sin(o + depth[:, None] * d + which[:, None])
    return depth.view(height, width).contiguous(), color.view(height, width, 3).contiguous()


def _room_frames(case, g):
    """A recording that sees the room once around: one pose per direction of a spherical lattice."""
    room, n, H, W = _room(g), case["frames"], case["height"], case["width"]
    focal = 525.0 * W / 640.0
    K = torch.tensor([[focal, 0.0, (W - 1) / 2.0], [0.0, focal, (H - 1) / 2.0], [0.0, 0.0, 1.0]])
    jitter = ((torch.rand(n, 2, 3, generator=g, device=DEVICE) - 0.5) * 0.8).double().cpu()
    turn = float(torch.rand(1, generator=g, device=DEVICE))
    frames = []
    for i in range(n):
        z = 1.0 - 2.0 * (i + 0.5) / n
        phi = math.pi * (3.0 - math.sqrt(5.0)) * (i + 0.5) + 2 * math.pi * turn
        way = torch.tensor([math.sqrt(1 - z * z) * math.cos(phi), math.sqrt(1 - z * z) * math.sin(phi), z], dtype=torch.float64)
        wall = way * (5.0 / way.abs().max())
        pose = _camera((wall - 3.2 * way + jitter[i, 0]).clamp(-4.2, 4.2), wall + jitter[i, 1])
        depth, color = _room_frame(room, K, pose, H, W)
        frames.append(ash.DotDict(depth=depth, depth_scale=1.0, depth_max=5.0, intrinsic=K.numpy(),
                                  extrinsic=torch.linalg.inv(pose).numpy(), rgb=color))
    return frames


def _prepare_fuse(case, g):
    frames = _room_frames(case, g)

    def volume(capacity):
        return ash.UnBoundedSparseDenseGrid(3, capacity, 5, 8, cell_size=case["voxel"], device=DEVICE)

    n = _reached(case)
    grid = volume(2 * n)
    TSDFFusion(grid, case["dilation"]).fuse_dataset(frames)
    blocks = grid.engine.items()[0]
    x, y, z = (blocks[:, i].long() + 2**20 for i in range(3))
    blocks = blocks[torch.argsort((x << 42) + (y << 21) + z)].contiguous()     # the blocks that the recording reaches, in order
    grid = volume(n)
    if case["frames"] == 1:                     # a volume that holds them already
        _load_blocks(grid, blocks[:n])
    blocks = blocks[torch.arange(n, device=DEVICE) % blocks.shape[0]].contiguous()   # some twice: as many for every seed
    return {"grid": grid, "fusion": TSDFFusion(grid, case["dilation"]), "frames": frames, "blocks": blocks}


def _run_fuse(s):
    grid, frames = s["grid"], s["frames"]
    if len(frames) == 1:
        s["fusion"].fuse_frame(frames[0])
        return grid.embeddings.data
    grid.engine.clear()
    grid.embeddings.data.zero_()
    s["fusion"].fuse_dataset(frames)
    rows, masks = grid.engine.find(s["blocks"])     # the volume block by block, in a fixed order
    return grid.embeddings.data[rows], masks


def _seen(case):
    """Blocks within reach of the surfaces that one frame sees, on average."""
    return 3_500 * (0.015 / case["voxel"]) ** 2 * (1.0 if case["dilation"] == 1 else 1.7)


def _reached(case):
    """Somewhat more blocks than the whole recording reaches."""
    room = 160_000 * (0.015 / case["voxel"]) ** 2 * (1.0 if case["dilation"] == 1 else 1.7)
    return int(min(room, 4 * case["frames"] * _seen(case)))


def _work_fuse(case):
    block = 512 * 5 * 4
    images = case["frames"] * case["height"] * case["width"] * 16
    volume = 3 * _reached(case) * block if case["frames"] > 1 else 0     # emptied before, read and written after
    return {"bytes": images + case["frames"] * _seen(case) * 2 * block + volume, "flops": case["frames"] * _seen(case) * 512 * 50}


# ----------------------------------------------------------------------------------------- mesh
def _prepare_mesh(case, g):
    room, G = _room(g), case["grid_dim"]
    blocks, side = _room_blocks(case["blocks"], room, g)
    blocks = blocks - side // 2
    cell = 2.0 / (side * G)
    grid = ash.UnBoundedSparseDenseGrid(3, blocks.shape[0], 1, G, cell_size=cell, device=DEVICE)
    _load_blocks(grid, blocks)
    grid.construct_grid_neighbor_lut_(radius=1, bidirectional=False)
    shift = 0.2 * cell * torch.rand(3, generator=g, device=DEVICE)
    tsdf = torch.empty(blocks.shape[0], G**3, device=DEVICE)
    weight = torch.empty_like(tsdf)
    for at in range(0, blocks.shape[0], 4096):      # the field in pieces: it is evaluated sphere by sphere
        p = ((blocks[at:at + 4096, None, :] * G + grid.cell_coords[None]).float() + 0.01) * cell + shift
        d = _room_distance(room, p) + 0.1 * cell * torch.sin(40.0 * p).sum(-1)
        tsdf[at:at + 4096] = d.clamp(-4 * G * cell, 4 * G * cell)
        weight[at:at + 4096] = (p[..., 0] + 0.5 * p[..., 1] < 0.9).float() * 3.0     # a corner was never observed
    most = 2 * _vertices(case)
    return {"grid": grid, "tsdf": tsdf, "weight": weight, "vertices": torch.zeros(most, 3, device=DEVICE),
            "triangles": torch.zeros(2 * most, dtype=torch.long, device=DEVICE)}


def _run_mesh(s):
    surface = s["grid"].marching_cubes(s["tsdf"], s["weight"], vertices_only=False)
    p, t = surface["positions"], surface["triangles"].long()
    # Vertices and triangles come in no defined order; put them in one.
    bits = p.contiguous().view(torch.int32).long()
    key, order = torch.sort((bits[:, 0] * 0x2545F4914F6CDD1D + bits[:, 1]) * 0x27BB2EE687B0B0FD + bits[:, 2])
    name = torch.empty_like(order)
    name[order] = torch.cumsum(torch.cat([key.new_zeros(1), (key[1:] != key[:-1]).long()]), 0)
    t = name[t]
    first = t.argmin(dim=1, keepdim=True)
    a, b, c = (t.gather(1, (first + k) % 3)[:, 0] for k in range(3))
    n = p.shape[0]
    vertices, triangles = s["vertices"].zero_(), s["triangles"].fill_(-1)     # of one size for every surface
    vertices[:n], triangles[: t.shape[0]] = p[order], torch.sort((a * n + b) * n + c)[0]
    return vertices, triangles, n, t.shape[0]


def _vertices(case):
    return int(60 * case["blocks"] * (case["grid_dim"] / 8) ** 2) + 1_000


def _work_mesh(case):
    cells = case["blocks"] * case["grid_dim"] ** 3
    return {"bytes": cells * 8 + 3 * 12 * _vertices(case), "flops": cells * 10}


# ----------------------------------------------------------------------------------------- smooth
def _prepare_smooth(case, g):
    grid, _ = _room_grid(case, g)
    grid.embeddings.data.normal_(0, 0.1, generator=g)
    return {"grid": grid, "size": case["size"]}


def _run_smooth(s):
    s["grid"].gaussian_filter_(s["size"], 1.0)
    return s["grid"].embeddings.data


def _work_smooth(case):
    row = case["grid_dim"] ** 3 * case["channels"] * 4
    spare = max(0, case["capacity"] - case["blocks"])   # rows without a block come out as zeros
    return {"bytes": (2 * case["blocks"] + spare) * row, "flops": case["blocks"] * row / 4 * 6 * case["size"]}


# ----------------------------------------------------------------------------------------- render
def _prepare_render(case, g):
    grid, room = _room_grid(case, g)
    blocks = grid.engine.items()
    with torch.no_grad():
        grid.embeddings.normal_(0, 0.02, generator=g)
        coords, rows = blocks
        for at in range(0, rows.shape[0], 4096):
            p = grid.cell_to_world(coords[at:at + 4096], grid.cell_coords).view(-1, grid.num_cells_per_grid, 3)
            cells = grid.embeddings[rows[at:at + 4096]]
            cells[..., 0] = _room_distance(room, p) + 0.02 * grid.cell_size * cells[..., 0]
            cells[..., 1:4] += 0.5 + 0.5 * torch.sin(7.0 * p)
            grid.embeddings[rows[at:at + 4096]] = cells
    n = case["rays"]
    if case["train"]:       # pixels of many views
        o = (torch.rand(n, 3, generator=g, device=DEVICE) - 0.5) * 1.2
        to = (torch.rand(n, 3, generator=g, device=DEVICE) - 0.5) * 1.2
        d = to - o
    else:                   # the pixels of one view, row by row
        width = max(1, int(math.sqrt(n * 4 / 3)))
        pixel = torch.arange(n, device=DEVICE)
        u, v = (pixel % width + 0.5) / width - 0.5, (torch.div(pixel, width, rounding_mode="floor") + 0.5) / width - 0.375
        turn = 2 * math.pi * float(torch.rand(1, generator=g, device=DEVICE))
        along = torch.stack([math.cos(turn) - 1.2 * u * math.sin(turn), math.sin(turn) + 1.2 * u * math.cos(turn), -1.2 * v], -1)
        o = ((torch.rand(1, 3, generator=g, device=DEVICE) - 0.5) * 0.6).repeat(n, 1)
        d = along
    grid.construct_grid_neighbor_lut_(radius=1, bidirectional=False)
    to_density = SDFToDensity(min_beta=grid.cell_size, init_beta=2 * grid.cell_size).to(DEVICE)
    target = torch.rand(n, 3, generator=g, device=DEVICE)
    return {"grid": grid, "to_density": to_density, "o": o.contiguous(), "d": torch.nn.functional.normalize(d, dim=-1).contiguous(),
            "target": target, "samples": case["samples"], "interpolation": case["interpolation"], "train": case["train"]}


def _run_render(s):
    grid, module = s["grid"], s["to_density"]
    if not s["train"]:
        with torch.no_grad():
            beta = module.min_beta + module.beta.abs()
            view = render_rays(grid, s["o"], s["d"], 0.06, 2.5, s["samples"], beta, s["interpolation"], skip_rays_without_hit=True)
        return view["rgb"], view["depth"], view["normal"], view["weights"], view["n_samples"]
    grid.embeddings.grad = None
    module.beta.grad = None
    beta = module.min_beta + module.beta.abs()
    out = render_rays(grid, s["o"], s["d"], 0.06, 2.5, s["samples"], beta, s["interpolation"], skip_rays_without_hit=True)
    loss = (out["rgb"] - s["target"]).abs().mean() + 0.1 * (out["depth"] - 0.3).abs().mean() \
        + 0.1 * out["eikonal_l2"].sum() / out["n_samples"].sum().clamp_min(1)
    loss.backward()
    return out["rgb"].detach(), out["depth"].detach(), grid.embeddings.grad, module.beta.grad


def _work_render(case):
    samples = 12 * case["rays"]
    row = 512 * case["channels"] * 4
    touched = min(case["blocks"] * row, samples * 8 * 16)
    work = {"bytes": case["rays"] * (24 + 13 * 4) + touched, "flops": samples * 200}
    if case["train"]:
        work = {"bytes": 2 * work["bytes"] + max(case["capacity"], case["blocks"]) * row, "flops": 3 * work["flops"]}
    return work


# ----------------------------------------------------------------------------------------- the interface
_KINDS = {"hash": (_prepare_hash, _run_hash, _work_hash), "query": (_prepare_query, _run_query, _work_query),
          "eikonal": (_prepare_query, _run_eikonal, _work_query), "fuse": (_prepare_fuse, _run_fuse, _work_fuse),
          "mesh": (_prepare_mesh, _run_mesh, _work_mesh), "smooth": (_prepare_smooth, _run_smooth, _work_smooth),
          "render": (_prepare_render, _run_render, _work_render)}


def prepare(case, seed):
    return {"kind": case["kind"], **_KINDS[case["kind"]][0](case, _generator(seed))}


def run(state):
    return _KINDS[state["kind"]][1](state)


def work(case):
    return _KINDS[case["kind"]][2](case)


def tolerance(case):
    """About four times what was seen between two correct orders of the sums (float64 tables, the tiled instead of the
    separable filter, rays marched by one thread instead of a warp).  "max" is wider where single rows cancel."""
    return {"hash": "exact", "query": {"rel": 1e-6, "max": 4e-5}, "eikonal": {"rel": 1e-6, "max": 5e-4}, "fuse": "exact",
            "mesh": "exact", "smooth": {"rel": 1.5e-6, "max": 2e-5}, "render": {"rel": 4e-6, "max": 8e-3}}[case["kind"]]
