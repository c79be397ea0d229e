"""The work that a user of this framework has it do, as cases to be timed.

Each case is one call, or one chain of calls, of the public entry points
(``triangle_extraction``, ``triangle_rasterization``, ``subdivision``,
``graph``), at sizes of the repository's own configurations
(``synthetic.CONFIGS``), of its benchmark and of its tests. ``kind`` says
which:

``step``         a training step called as a trainer calls it: tessellate,
                 render, mean squared error, backward into the grid
``captured``     the same step replayed as one CUDA graph
``tessellate``   marching cubes of every shell, forward and backward
``render``       a batch of cameras of one size, forward and backward
``cameras``      a batch of cameras of different sizes, forward and backward
``view``         one image of a resident mesh, no gradient
``extract``      a packed occupancy grid to its sparse voxel topology
``subdivide``    a scene's parameters onto a finer grid
``regularizers`` the SDF losses, forward and backward

Scenes are unions of spheres in a sparse voxel band, as the benchmark's. The
seed draws the signed distances (each between the two level sets that it lies
between, so that a case's sizes are those of every seed), the colours, the
camera positions, the targets and the gradients that come from outside; of an
occupancy grid, where in its box the scene lies and which way it faces.
"""

from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from meshtryoshka_gb300 import graph, pipeline, subdivision, synthetic
from meshtryoshka_gb300 import triangle_extraction as te
from meshtryoshka_gb300 import triangle_rasterization as tr

# Sphere layouts: the 64^3 test sphere, the benchmark's eight spheres, and the
# large configuration's spheres inside a background sphere.
LAYOUTS = {"one": "small", "eight": "mid", "room": "large"}


def _scene(i, j, k, layout, shells, span, sh_degree, band=2.0):
    return {"i": i, "j": j, "k": k, "layout": layout, "band": band, "shells": shells, "span": span,
            "sh_degree": sh_degree}


def _shots(rig, count, height, width, fov=50.0):
    return {"rig": rig, "cameras": count, "height": height, "width": width, "fov": fov}


def listed():
    mid = _scene(256, 256, 256, "eight", 8, 0.03, 3)
    large = _scene(512, 512, 512, "room", 16, 0.02, 3)
    return [
        # The first stage of a coarse-to-fine run, and every debugging session:
        # a few thousand voxels, one small image, colours without view
        # dependence. Launches and host work count.
        {"name": "step_64_one_128", "kind": "step", **_scene(64, 64, 64, "one", 3, 0.02, 0),
         **_shots("front", 1, 128, 128, 60.0), "mode": "fused"},
        # The benchmark's headline step (256^3, 8 shells, 4 x 800^2) as a
        # training loop runs it, captured, at the tile shape the autotuner
        # picks for it.
        {"name": "captured_256_mid", "kind": "captured", **mid, **_shots("orbit", 4, 800, 800),
         "tile_h": 8, "tile_w": 8, "threads": 256},
        # The last stage of training a room-sized scene: 512^3, 16 shells,
        # cameras inside the scene with an odd image width.
        {"name": "captured_512_room", "kind": "captured", **large, **_shots("ring", 4, 840, 1297, 55.0),
         "tile_h": 16, "tile_w": 8, "threads": 256},
        # The tessellation half of a trainer's step at the large grid, with
        # the default arguments: per-vertex coefficient rows formed, and
        # their gradient sent back to the grid.
        {"name": "tessellate_512_room", "kind": "tessellate", **_scene(512, 512, 512, "room", 8, 0.02, 3)},
        # The rendering half of a trainer's step with the default arguments,
        # in the fused mode and in the explicit mode.
        {"name": "render_mid_fused", "kind": "render", **mid, **_shots("orbit", 4, 800, 800), "mode": "fused",
         "ssaa": 1},
        {"name": "render_mid_explicit", "kind": "render", **mid, **_shots("orbit", 4, 800, 800), "mode": "explicit",
         "ssaa": 1},
        # A capture whose photographs differ in size, trained on as one batch.
        {"name": "cameras_mid_uneven", "kind": "cameras", **mid, "rig": "orbit", "cameras": 32, "shapes": 2,
         "least": 200, "most": 1600, "fov": 55.0},
        # A viewer's frame, and a served request: one small image of a
        # resident mesh.
        {"name": "view_mid_256", "kind": "view", **mid, **_shots("orbit", 1, 256, 256), "ssaa": 1},
        # A still for a figure: full HD, two by two samples to a pixel.
        {"name": "view_mid_1080_ssaa", "kind": "view", **mid, **_shots("orbit", 1, 1080, 1920), "ssaa": 2},
        # The topology of a new grid, after each subdivision and when a
        # checkpoint is loaded.
        {"name": "extract_512_room", "kind": "extract", **_scene(512, 512, 512, "room", 1, 0.0, 0)},
        # The subdivision between two stages of training.
        {"name": "subdivide_mid_512", "kind": "subdivide", **mid, "to_i": 512, "to_j": 512, "to_k": 512},
        # The losses on the grid itself, taken beside every step.
        {"name": "regularizers_512_room", "kind": "regularizers", **_scene(512, 512, 512, "room", 1, 0.0, 0)},
    ]


def _spread(rng, low, high):
    """A whole number, even in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "captured", "tessellate", "render", "render", "cameras", "view", "extract",
                       "subdivide", "regularizers"])
    layout = rng.choice(["one", "eight", "eight", "room"])
    most = {"one": 512, "eight": 480, "room": 352}[layout]
    if kind == "subdivide":
        most = 256
    side = _spread(rng, 48, most)
    # Grids are boxes: any extents, the packed axis in whole words.
    i, j = (max(33, side - rng.randrange(0, 14)) for _ in range(2))
    k = max(32, (side + 16) // 32 * 32)
    shells = rng.randint(1, 12)
    scene = _scene(i, j, k, layout, shells, 0.0 if shells == 1 else rng.uniform(0.005, 0.03), rng.randint(0, 3))
    rig = {"one": "front", "eight": "orbit", "room": "ring"}[layout]
    case = {"kind": kind, **scene}
    if kind in ("step", "captured", "render", "view"):
        ssaa = rng.choice([1, 1, 2]) if kind in ("render", "view") else 1
        pixels = _spread(rng, 100 * 100, (2000 if kind == "view" else 1100) ** 2 // ssaa**2)
        height = max(64, int(math.sqrt(pixels * rng.uniform(0.5, 1.6))))
        width = max(64, pixels // height)
        count = 1 if kind == "view" or rig == "front" else max(1, min(rng.randint(1, 6), 4_500_000 // (pixels * ssaa**2)))
        case.update(_shots(rig, count, height, width, rng.uniform(40.0, 70.0)))
        if kind == "captured":
            case["tile_h"], case["tile_w"] = rng.choice([(8, 8), (16, 8), (16, 16)])
            case["threads"] = 256
        if kind in ("step", "render"):
            case["mode"] = rng.choice(["fused", "fused", "explicit"])
        if kind in ("render", "view"):
            case["ssaa"] = ssaa
    elif kind == "cameras":
        low = rng.randint(64, 300)
        case.update(rig=rig, cameras=rng.randint(2, 16), shapes=rng.randrange(1 << 16), least=low,
                    most=low + rng.randint(50, 900), fov=rng.uniform(40.0, 70.0))
    elif kind == "subdivide":
        grow = rng.uniform(1.0, 2.0)
        case.update(to_i=int(i * grow), to_j=int(j * grow), to_k=int(math.ceil(k * grow / 32)) * 32)
    return case


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _config(case):
    base = synthetic.CONFIGS[LAYOUTS[case["layout"]]]
    span, n = case["span"], case["shells"]
    levels = tuple(span - 2.0 * span * s / max(n - 1, 1) for s in range(n)) if n > 1 else (0.0,)
    return dataclasses.replace(base, sh_degree=case["sh_degree"], level_sets=levels, band_voxels=case["band"])


def _spheres(cfg, device):
    centres, radii = synthetic.sphere_layout(cfg)
    return torch.from_numpy(centres).to(device), torch.from_numpy(radii).to(device)


def _packed(occupied):
    n_i, n_j, n_k = occupied.shape
    powers = 1 << torch.arange(32, device=occupied.device, dtype=torch.int64)
    words = (occupied.reshape(n_i, n_j, n_k // 32, 32) * powers).sum(-1)
    return words.to(torch.uint32).view(torch.int32)


def _unpacked(packed):
    bits = torch.arange(32, device=packed.device, dtype=torch.int32)
    return ((packed[..., None] >> bits) & 1).flatten(-2).bool()


def _occupancy(case, cfg, spheres):
    """Packed occupancy of the band around the surface, in slabs along i."""
    n_i, n_j, n_k = case["i"], case["j"], case["k"]
    device = spheres[0].device
    axis = [2.0 * (torch.arange(n, device=device, dtype=torch.float32) + 0.5) / n - 1.0 for n in (n_i, n_j, n_k)]
    packed = torch.empty((n_i, n_j, n_k // 32), dtype=torch.int32, device=device)
    slab = max(1, (1 << 24) // (n_j * n_k))
    for at in range(0, n_i, slab):
        z, y, x = torch.meshgrid(axis[0][at:at + slab], axis[1], axis[2], indexing="ij")
        d = synthetic.analytic_sdf(torch.stack((x, y, z), dim=-1), *spheres, cfg.background_radius)
        packed[at:at + slab] = _packed(d.abs() < cfg.band_voxels * 2.0 / n_k)
    return packed


def _turned(occupancy, seed):
    """The same scene facing another way and, where its box has room along i and j, elsewhere in it."""
    occupied = _unpacked(occupancy)
    occupied = occupied.flip([a for a in range(3) if (seed >> a) & 1])
    rng = np.random.default_rng(seed)
    for axis in (0, 1):
        rows = occupied.any(dim=2).any(dim=1 - axis).nonzero()[:, 0]
        if rows.numel():
            low, high = int(rows[0]), occupied.shape[axis] - 1 - int(rows[-1])
            occupied = occupied.roll(int(rng.integers(-min(low, 16), min(high, 16) + 1)), axis)
    return _packed(occupied)


def _redrawn(d, levels, rng):
    """Other signed distances that lie between the same two level sets: part of the way to one of the two."""
    edges = levels.sort()[0]
    edges = torch.cat((edges[:1] - 1.0, edges, edges[-1:] + 1.0))
    at = torch.searchsorted(edges, d.clamp(edges[0], edges[-1]), right=True).clamp(1, edges.numel() - 1)
    low, high = edges[at - 1], edges[at]
    part = torch.rand(d.shape, generator=rng, device=d.device) * 0.3
    up = torch.rand(d.shape, generator=rng, device=d.device) < 0.5
    # Near the ends of the range there is no level set to go to: a step of the noise's size.
    room = torch.where(up, high - d, low - d).clamp(-0.005, 0.005)
    new = d + part * room
    return torch.where((new >= low) & (new < high), new, d)


def _grid(case, seed):
    """Voxels, signed distances and coefficients of a scene."""
    device = _device()
    cfg = _config(case)
    spheres = _spheres(cfg, device)
    occupancy = _occupancy(case, cfg, spheres)
    voxels = te.extract_voxels(occupancy)
    levels = torch.tensor(cfg.level_sets, dtype=torch.float32, device=device)
    d = synthetic.analytic_sdf(2.0 * voxels.vertices - 1.0, *spheres, cfg.background_radius)
    d = d + cfg.noise_sigma * torch.randn(d.shape, generator=torch.Generator(device).manual_seed(0), device=device)
    rng = torch.Generator(device).manual_seed(seed)
    sdf = _redrawn(d, levels, rng)
    sh = 0.05 * torch.randn(((cfg.sh_degree + 1) ** 2, d.shape[0], 3), generator=rng, device=device)
    sh[0] = torch.rand(sh[0].shape, generator=rng, device=device)
    return {"config": cfg, "occupancy": occupancy, "voxels": voxels, "sdf": sdf.contiguous(), "sh": sh,
            "levels": levels, "sharpness": torch.tensor(cfg.sharpness, device=device),
            "background": torch.tensor((0.1, 0.2, 0.3), device=device), "rng": rng}


def _eye(rig, index, count, rng):
    if rig == "front":
        return 2.0 * np.array([rng.uniform(-0.05, 0.05), rng.uniform(-0.05, 0.05), 1.0])
    if rig == "orbit":
        # Around the scene, evenly spread, so that a scene's cameras see alike
        # much of it whatever the seed.
        az = 2.0 * math.pi * (index + rng.uniform(0.2, 0.4)) / count
        el = math.radians(rng.uniform(30.0, 40.0))
        return 2.5 * np.array([math.cos(el) * math.cos(az), math.sin(el), math.cos(el) * math.sin(az)])
    az = 2.0 * math.pi * (index + rng.uniform(0.0, 0.1)) / count
    return 0.6 * np.array([math.cos(az), 0.0, math.sin(az)])


def _image_shapes(case):
    if "shapes" in case:
        rng = np.random.default_rng(case["shapes"])
        return [tuple(int(x) for x in rng.integers(case["least"], case["most"] + 1, 2)) for _ in range(case["cameras"])]
    return [(case["height"], case["width"])] * case["cameras"]


def _cameras(case, seed):
    device, rng = _device(), np.random.default_rng(seed)
    shapes = _image_shapes(case)
    ext = [synthetic.look_at(_eye(case["rig"], b, len(shapes), rng)) for b in range(len(shapes))]
    intr = [synthetic.pinhole(h, w, case["fov"]) for h, w in shapes]
    return {"extrinsics": torch.from_numpy(np.stack(ext)).to(device),
            "intrinsics": torch.from_numpy(np.stack(intr)).to(device), "shapes": shapes}


def _tessellated(s, **kw):
    v = s["voxels"]
    return te.tessellate_voxels(s["sdf"], v.vertices, s["sh"], v.neighbors, v.lower_corners, v.upper_corners,
                                v.indices, s["levels"], **kw)


def prepare(case, seed):
    device, kind = _device(), case["kind"]
    if kind == "extract":
        cfg = _config(case)
        occupancy = _turned(_occupancy(case, cfg, _spheres(cfg, device)), seed)
        return {"kind": kind, "case": case, "occupancy": occupancy}
    s = _grid(case, seed)
    s.update(kind=kind, case=case)
    if kind in ("step", "captured", "render", "cameras", "view"):
        s.update(_cameras(case, seed))
        s["targets"] = [torch.rand((3, h, w), generator=s["rng"], device=device) for h, w in s["shapes"]]
    if kind == "step":
        s["target"] = torch.stack(s["targets"])
        s["sdf"].requires_grad_(True)
        s["sh"].requires_grad_(True)
    elif kind == "captured":
        s["step"] = graph.CapturedTrainingStep(pipeline.Workload(
            config=s["config"], voxels=s["voxels"], grid_sdf=s["sdf"].requires_grad_(True),
            grid_sh=s["sh"].requires_grad_(True), level_sets=s["levels"], extrinsics=s["extrinsics"],
            intrinsics=s["intrinsics"], image_shape=s["shapes"][0], target=torch.stack(s["targets"]),
            sharpness=s["sharpness"], background=s["background"],
            tile_shape=(case["tile_h"], case["tile_w"], case["threads"])))
    elif kind == "tessellate":
        with torch.no_grad():
            tri = _tessellated(s)
        s["grad_vertex_sdf"] = torch.randn(tri.signed_distances.shape, generator=s["rng"], device=device)
        s["grad_vertex_sh"] = torch.randn(tri.spherical_harmonics.shape, generator=s["rng"], device=device)
        s["sdf"].requires_grad_(True)
        s["sh"].requires_grad_(True)
    elif kind in ("render", "cameras", "view"):
        with torch.no_grad():
            tri = _tessellated(s)
        s.update(vertices=2.0 * tri.vertices - 1.0, faces=tri.faces, boundaries=tri.face_boundaries,
                 vertex_sdf=tri.signed_distances.clone(), vertex_sh=tri.spherical_harmonics.clone())
        if kind == "render":
            s["target"] = torch.stack(s["targets"])
        if kind != "view":
            s["vertex_sdf"].requires_grad_(True)
            s["vertex_sh"].requires_grad_(True)
    elif kind == "subdivide":
        with torch.no_grad():
            s["triangle_voxels"] = _tessellated(s).voxel_indices
    elif kind == "regularizers":
        s["sdf"].requires_grad_(True)
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _render(s, **kw):
    return tr.render(s["extrinsics"], s["intrinsics"], s["shapes"][0], s["vertices"], s["faces"], s["boundaries"],
                     s["vertex_sdf"], s["vertex_sh"], s["config"].sh_degree, s["sharpness"], s["background"], **kw)


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "step":
        tri = _tessellated(s)
        vertices = (2.0 * tri.vertices - 1.0).detach()
        images = tr.render(s["extrinsics"], s["intrinsics"], s["shapes"][0], vertices, tri.faces, tri.face_boundaries,
                           tri.signed_distances, tri.spherical_harmonics, case["sh_degree"], s["sharpness"],
                           s["background"], mode=case["mode"])
        loss = ((images - s["target"]) ** 2).mean()
        grad_sdf, grad_sh = torch.autograd.grad(loss, (s["sdf"], s["sh"]))
        return {"images": images.detach(), "loss": loss.detach(), "grad_sdf": grad_sdf, "grad_sh": grad_sh}
    if kind == "captured":
        step = s["step"]
        loss = step()
        return {"loss": loss, "grad_sdf": step.grad_sdf, "grad_sh": step.grad_sh}
    if kind == "tessellate":
        tri = _tessellated(s)
        grad_sdf, grad_sh = torch.autograd.grad((tri.signed_distances, tri.spherical_harmonics), (s["sdf"], s["sh"]),
                                                (s["grad_vertex_sdf"], s["grad_vertex_sh"]))
        return {**{k: v.detach() for k, v in tri._asdict().items()}, "grad_sdf": grad_sdf, "grad_sh": grad_sh}
    if kind == "render":
        images = _render(s, mode=case["mode"], ssaa=case["ssaa"])
        loss = ((images - s["target"]) ** 2).mean()
        grad_sdf, grad_sh = torch.autograd.grad(loss, (s["vertex_sdf"], s["vertex_sh"]))
        return {"images": images.detach(), "loss": loss.detach(), "grad_sdf": grad_sdf, "grad_sh": grad_sh}
    if kind == "cameras":
        images = tr.render_cameras(s["extrinsics"], s["intrinsics"], s["shapes"], s["vertices"], s["faces"],
                                   s["boundaries"], s["vertex_sdf"], s["vertex_sh"], case["sh_degree"],
                                   s["sharpness"], s["background"])
        loss = sum(((a - b) ** 2).sum() for a, b in zip(images, s["targets"])) / sum(3 * h * w for h, w in s["shapes"])
        grad_sdf, grad_sh = torch.autograd.grad(loss, (s["vertex_sdf"], s["vertex_sh"]))
        return {"images": [x.detach() for x in images], "loss": loss.detach(), "grad_sdf": grad_sdf,
                "grad_sh": grad_sh}
    if kind == "view":
        with torch.no_grad():
            return {"images": _render(s, ssaa=case["ssaa"])}
    if kind == "extract":
        return list(te.extract_voxels(s["occupancy"])[:5])
    if kind == "subdivide":
        return list(subdivision.subdivide(s["voxels"], s["sdf"], s["sh"], s["occupancy"], s["triangle_voxels"],
                                          (case["to_i"], case["to_j"], case["to_k"])))
    v = s["voxels"]
    losses = te.compute_sdf_regularizers(s["sdf"], v.neighbors, v.lower_corners, v.upper_corners, v.grid_shape)
    total = losses.eikonal_loss_pos.mean() + losses.eikonal_loss_neg.mean() + 10.0 * losses.curvature_loss.mean()
    (grad_sdf,) = torch.autograd.grad(total, (s["sdf"],))
    return {**{k: v.detach() for k, v in losses._asdict().items()}, "grad_sdf": grad_sdf}


def _size(values):
    """Bytes of the tensors among (nested) values."""
    if isinstance(values, torch.Tensor):
        return values.numel() * values.element_size()
    if isinstance(values, dict):
        values = list(values.values())
    return sum(_size(v) for v in values) if isinstance(values, (list, tuple)) else 0


def work(case):
    """The bytes of one pass's inputs and outputs, from a scene of the case;
    what is formed in between is not counted. The arithmetic is small beside
    them."""
    s = prepare(case, 0)
    used = {"step": ("sdf", "sh", "voxels", "levels", "extrinsics", "intrinsics", "targets"),
            "tessellate": ("sdf", "sh", "voxels", "levels", "grad_vertex_sdf", "grad_vertex_sh"),
            "view": ("vertices", "faces", "vertex_sdf", "vertex_sh", "extrinsics", "intrinsics"),
            "extract": ("occupancy",),
            "subdivide": ("voxels", "sdf", "sh", "occupancy", "triangle_voxels"),
            "regularizers": ("sdf",)}
    used["captured"] = used["step"]
    used["render"] = used["cameras"] = used["view"] + ("targets",)
    moved = _size([s[k] for k in used[s["kind"]]]) + _size(run(s))
    if s["kind"] == "subdivide":  # of the topology, only the vertices
        moved -= _size([v for k, v in s["voxels"]._asdict().items() if k != "vertices"])
    if s["kind"] == "regularizers":  # the corners, and the +xyz neighbours
        v = s["voxels"]
        moved += _size([v.lower_corners, v.upper_corners]) + 4 * v.num_voxels
    return {"bytes": float(moved), "flops": 0.0}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
#
# Whole numbers and decisions (which triangles a pixel meets, in which order)
# are made in the 32 bits that define them, operation by operation; every
# value is then computed in 64 bits. Gradients follow the routing of the
# default gradient mode: a hit's deferred gradient goes to its own triangle
# with the weights of the next hit (fused), or the signed-distance part to
# the slot before the next hit's shell (explicit).
# ---------------------------------------------------------------------------
NEAR = 0.2
MOST_FACES = 8_000_000  # faces x cameras above which the 64-bit image takes too long


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "captured"):
        return None  # whole calls: their halves have cases of their own
    s = prepare(case, seed)
    with torch.no_grad():
        if kind == "extract":
            return [_exact_vertices(s["occupancy"]), None, None, None, None]
        if kind == "subdivide":
            return _exact_subdivision(s, (case["to_i"], case["to_j"], case["to_k"]))
        if kind == "tessellate":
            return _exact_tessellation(s)
        if kind in ("render", "cameras", "view"):
            if s["faces"].shape[0] * len(s["shapes"]) > MOST_FACES and kind != "cameras":
                return None
            return _exact_render(s, kind)
    return _exact_regularizers(s)


def _corner_points(occupied):
    """Grid points that are a corner of an occupied voxel."""
    i, j, k = occupied.shape
    points = torch.zeros((i + 1, j + 1, k + 1), dtype=torch.bool, device=occupied.device)
    for a in range(8):
        x, y, z = a >> 2, (a >> 1) & 1, a & 1
        points[x:x + i, y:y + j, z:z + k] |= occupied
    return points


def _exact_vertices(occupancy):
    occupied = _unpacked(occupancy)
    at = _corner_points(occupied).nonzero().flip(-1).double()  # (k, j, i)
    return at / torch.tensor(occupied.shape[::-1], device=at.device, dtype=torch.float64)


def _exact_subdivision(s, target):
    old = _unpacked(s["occupancy"])
    device = old.device
    touched = torch.zeros(old.numel(), dtype=torch.bool, device=device)
    touched[s["triangle_voxels"].long()] = True
    near = touched.reshape(old.shape)
    for axis in range(3):  # a box of four voxels to each side
        n = near.shape[axis]
        near = torch.stack([torch.nn.functional.pad(near.movedim(axis, 0).float(), (0, 0, 0, 0, 4, 4))[d:d + n]
                            for d in range(9)]).amax(0).movedim(0, axis) > 0
    kept = old & near
    sides = []
    for n_old, n_new in zip(old.shape, target):
        at = torch.arange(n_new, device=device)
        sides.append(((at * n_old) // n_new, ((at + 1) * n_old - 1) // n_new))
    grown = torch.zeros(target, dtype=torch.bool, device=device)
    for a in range(8):
        pick = [sides[axis][(a >> axis) & 1] for axis in range(3)]
        grown |= kept[pick[0]][:, pick[1]][:, :, pick[2]]
    old_points = _corner_points(old)
    ids = torch.full(old_points.shape, -1, dtype=torch.int64, device=device)
    ids[old_points] = torch.arange(int(old_points.sum()), device=device)
    at = _corner_points(grown).nonzero()
    scale = torch.tensor([a / b for a, b in zip(old.shape, target)], device=device, dtype=torch.float64)
    # The cell is the exact one: at * old // new.
    old_shape, new_shape = (torch.tensor(x, device=device) for x in (old.shape, target))
    cell = at * old_shape // new_shape
    part = at * scale - cell
    sdf, sh = s["sdf"].double(), s["sh"].double()
    new_sdf = torch.zeros(at.shape[0], dtype=torch.float64, device=device)
    new_sh = torch.zeros((sh.shape[0], at.shape[0], 3), dtype=torch.float64, device=device)
    total = torch.zeros_like(new_sdf)
    last = old_shape  # grid points run to the extent
    for q in range(8):
        d = torch.tensor([q >> 2, (q >> 1) & 1, q & 1], device=device)
        corner = cell + d
        inside = (corner <= last).all(1)
        index = torch.where(inside, ids[tuple(torch.minimum(corner, last).unbind(1))], -1)
        weight = torch.where(d.bool(), part, 1.0 - part).prod(1) * (index >= 0)
        index = index.clamp(min=0)
        total += weight
        new_sdf += weight * sdf[index]
        for c in range(sh.shape[0]):
            new_sh[c] += weight[:, None] * sh[c, index]
    return [new_sdf / total, new_sh / total[:, None], None]


def _exact_tessellation(s):
    sdf, sh, points = s["sdf"].double(), s["sh"].double(), s["voxels"].vertices.double()
    lower = s["voxels"].lower_corners.long()
    n, device = lower.shape[1], sdf.device
    out = {"vertices": [], "signed_distances": [], "spherical_harmonics": []}
    grad_sdf = torch.zeros_like(sdf)
    grad_sh = torch.zeros_like(sh)
    done = 0
    for level in s["levels"].double():
        d0 = sdf[lower[0]]
        across = torch.stack([(lower[a] >= 0) & ((d0 < level) != (sdf[lower[a].clamp(min=0)] < level))
                              for a in (1, 2, 3)], dim=1)
        entry, axis = across.nonzero(as_tuple=True)
        i0, i1 = lower[0][entry], lower.reshape(-1)[(axis + 1) * n + entry]
        a, b = sdf[i0], sdf[i1]
        t = torch.where(a == b, torch.full_like(a, 0.5), ((level - a) / (b - a)).clamp(0.0, 1.0))
        out["vertices"].append(points[i0] + t[:, None] * (points[i1] - points[i0]))
        out["signed_distances"].append(a + t * (b - a))
        out["spherical_harmonics"].append((sh[:, i0] + t[:, None] * (sh[:, i1] - sh[:, i0])).float())
        g, gs = (s[k][..., done:done + len(entry), :] if s[k].dim() > 1 else s[k][done:done + len(entry)]
                 for k in ("grad_vertex_sdf", "grad_vertex_sh"))
        grad_sdf.index_add_(0, i0, (1.0 - t) * g.double())
        grad_sdf.index_add_(0, i1, t * g.double())
        for c in range(sh.shape[0]):
            grad_sh[c].index_add_(0, i0, (1.0 - t)[:, None] * gs[c].double())
            grad_sh[c].index_add_(0, i1, t[:, None] * gs[c].double())
        done += len(entry)
    whole = {k: None for k in ("faces", "voxel_indices", "vertex_boundaries", "face_boundaries")}
    return {"vertices": torch.cat(out["vertices"]), "signed_distances": torch.cat(out["signed_distances"]),
            "spherical_harmonics": torch.cat(out["spherical_harmonics"], dim=1).double(), **whole,
            "grad_sdf": grad_sdf, "grad_sh": grad_sh}


def _exact_regularizers(s):
    v = s["voxels"]
    lower, upper, n = v.lower_corners.long(), v.upper_corners.long(), v.num_voxels
    sdf = s["sdf"].detach().double().requires_grad_(True)
    c000, c001, c010, c100 = (sdf[lower[r, :n]] for r in range(4))
    c111, c110, c101, c011 = (sdf[upper[r]] for r in range(4))
    i, j, k = v.grid_shape
    dx = 0.25 * k * (c001 - c000 + c011 - c010 + c101 - c100 + c111 - c110)
    dy = 0.25 * j * (c010 - c000 + c011 - c001 + c110 - c100 + c111 - c101)
    dz = 0.25 * i * (c100 - c000 + c101 - c001 + c110 - c010 + c111 - c011)
    delta = torch.sqrt(dx * dx + dy * dy + dz * dz) - 1.0
    pos, neg = delta.clamp(min=0.0) ** 2, delta.clamp(max=0.0) ** 2
    beyond = lower[1:, v.neighbors[6].long()]
    there = beyond >= 0
    around = c110 + c101 + c011 + (sdf[beyond.clamp(min=0)] * there).sum(0)
    curvature = (around - (3 + there.sum(0)) * c111) ** 2
    total = pos.mean() + neg.mean() + 10.0 * curvature.mean()
    (grad,) = torch.autograd.grad(total, (sdf,))
    return {"eikonal_loss_pos": pos.detach(), "eikonal_loss_neg": neg.detach(),
            "curvature_loss": curvature.detach(), "grad_sdf": grad}


def _basis(d, degree):
    """Real spherical harmonics at unit directions, by row."""
    x, y, z = d.unbind(1)
    rows = [torch.full_like(x, 0.28209479177387814)]
    if degree > 0:
        rows += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree > 1:
        rows += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
                 0.31539156525252005 * (2 * z * z - x * x - y * y), -1.0925484305920792 * x * z,
                 0.5462742152960396 * (x * x - y * y)]
    if degree > 2:
        rows += [-0.5900435899266435 * y * (3 * x * x - y * y), 2.890611442640554 * x * y * z,
                 -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
                 0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
                 -0.4570457994644658 * x * (4 * z * z - x * x - y * y), 1.445305721320277 * z * (x * x - y * y),
                 -0.5900435899266435 * x * (x * x - 3 * y * y)]
    return rows


def _project(vertices, ext, intr):
    """Pixel positions and depths, in the type of the arguments."""
    x, y, z = vertices.unbind(1)
    cam = [ext[r, 0] * x + ext[r, 1] * y + ext[r, 2] * z + ext[r, 3] for r in range(3)]
    px, py = ((intr[r, 0] * cam[0] + intr[r, 1] * cam[1] + intr[r, 2] * cam[2]) / cam[2] for r in range(2))
    return px, py, cam[2]


def _numerators(a, b, c, px, py):
    """Barycentric numerators (u, v, w) of pixels and their denominator."""
    e12, e13, e23 = ((q[0] - p[0], q[1] - p[1]) for p, q in ((a, b), (a, c), (b, c)))

    def dot(p, q):
        return p[0] * q[0] + p[1] * q[1]

    d1212, d1223, d1213, d1313, d1323, d2323 = (dot(p, q) for p, q in (
        (e12, e12), (e12, e23), (e12, e13), (e13, e13), (e13, e23), (e23, e23)))
    x, y, z = d1213.abs(), d1223.abs(), d1323.abs()
    den = torch.where((x <= y) & (x <= z), d1212 * d1313 - d1213 * d1213, torch.where(
        (y <= x) & (y <= z), d1212 * d2323 - d1223 * d1223, d1313 * d2323 - d1323 * d1323)) + 1e-8
    q1, q2 = (px - a[0], py - a[1]), (px - b[0], py - b[1])
    v = d1313 * dot(q1, e12) - d1213 * dot(q1, e13)
    w = d1212 * dot(q1, e13) - d1213 * dot(q1, e12)
    u = d1223 * dot(q2, e13) - d1323 * dot(q2, e12)
    return u / den, v / den, w / den


def _pixel_hits(s, camera, ext, intr, height, width):
    """(pixel, face, mean depth) of every accepted sample of a camera, faces in order."""
    faces = s["faces"].long()
    px, py, depth = _project(s["vertices"], ext, intr)
    a, b, c = ((px[f], py[f]) for f in faces.unbind(1))
    deep = depth[faces]
    facing = (b[0] - a[0]) * (c[1] - a[1]) - (b[1] - a[1]) * (c[0] - a[0])
    x = torch.stack((a[0], b[0], c[0]), 1)
    y = torch.stack((a[1], b[1], c[1]), 1)
    x0, x1 = x.amin(1).sub(1.5).clamp(0, width).int(), x.amax(1).add(1.5).clamp(0, width).int()
    y0, y1 = y.amin(1).sub(1.5).clamp(0, height).int(), y.amax(1).add(1.5).clamp(0, height).int()
    seen = ~(facing < 0) & ~(deep.amin(1) < NEAR) & (x1 > x0) & (y1 > y0)
    face = seen.nonzero()[:, 0]
    total = (deep[:, 0] + deep[:, 1]) + deep[:, 2]
    mean = total / torch.full_like(total, 3.0)  # a tensor: a number would be turned into its reciprocal
    found = []
    for part in face.split(1 << 18):
        wide = (x1 - x0)[part].long()
        many = wide * (y1 - y0)[part].long()
        which = torch.repeat_interleave(part, many)
        offset = torch.arange(which.shape[0], device=which.device) - torch.repeat_interleave(many.cumsum(0) - many, many)
        wide = torch.repeat_interleave(wide, many)
        row, col = y0[which] + offset // wide, x0[which] + offset % wide
        p = faces[which]
        u, v, w = _numerators(*((px[p[:, q]], py[p[:, q]]) for q in range(3)), col.float() + 0.5, row.float() + 0.5)
        total = u + v + w
        ok = (total >= 0.999) & (total <= 1.001)
        for q in (u, v, w):
            ok &= (q >= 0) & (q <= 1)
        found.append(torch.stack((row[ok].long() * width + col[ok], which[ok])))
    pixel, which = torch.cat(found, 1) if found else (face, face)
    return pixel, which, mean[which]


def _order(*keys):
    """Stable order by the last key, then the one before it, and so on."""
    at = torch.arange(keys[0].shape[0], device=keys[0].device)
    for key in keys:
        at = at[torch.sort(key[at], stable=True)[1]]
    return at


def _slots(pixel, face, depth, shell, shells, fused):
    """The samples that a pixel blends: [pixels with any], and per slot the face (-1: none).

    Fused: by depth, then shell, each deeper in the shells than the last; slots in that order.
    Explicit: the nearest sample of each shell; slots are shells."""
    at = _order(shell, depth, pixel) if fused else _order(depth, shell, pixel)
    pixel, face, shell = pixel[at], face[at], shell[at]
    which, inverse, many = torch.unique_consecutive(pixel, return_inverse=True, return_counts=True)
    slots = torch.full((which.shape[0], shells), -1, dtype=torch.int64, device=pixel.device)
    if not which.numel():
        return which, slots
    rank = torch.arange(pixel.shape[0], device=pixel.device) - (many.cumsum(0) - many)[inverse]
    last = torch.full_like(which, -1)
    used = torch.zeros_like(which)
    by_rank = torch.sort(rank, stable=True)[1].split(torch.bincount(rank).tolist())
    for at in by_rank:  # the r-th sample of every pixel
        to = inverse[at]
        ok = shell[at] > last[to]
        at, to = at[ok], to[ok]
        slots[to, used[to] if fused else shell[at]] = face[at]
        last[to] = shell[at]
        used[to] += 1
    return which, slots


def _exact_camera(s, camera, height, width, intr, fused, colors, dl):
    """A camera's [pixels, 4] composite (rgb, transmittance), and, given
    ``dl`` (a function of it: the loss's derivative), the gradients of the
    vertex colours and signed distances."""
    faces, shells = s["faces"].long(), s["boundaries"].shape[0]
    ext = s["extrinsics"][camera]
    pixel, face, depth = _pixel_hits(s, camera, ext, intr, height, width)
    shell = torch.searchsorted(s["boundaries"].long(), face, right=True)
    which, slots = _slots(pixel, face, depth, shell, shells, fused)
    image = torch.zeros((height * width, 4), dtype=torch.float64, device=faces.device)
    image[:, 3] = 1.0
    px, py, _ = _project(s["vertices"].double(), ext.double(), intr.double())
    sharp, sdf = s["sharpness"].double(), s["vertex_sdf"].detach().double()
    col, row = (which % width).double() + 0.5, (which // width).double() + 0.5
    there = slots >= 0
    corner = faces[slots.clamp(min=0)]  # [pixels, slots, 3]
    weight = torch.empty(corner.shape, dtype=torch.float64, device=faces.device)
    for l in range(shells):
        u, v, w = _numerators(*((px[corner[:, l, q]], py[corner[:, l, q]]) for q in range(3)), col, row)
        weight[:, l] = torch.stack((u, v, w if fused else 1.0 - u - v), 1)
    value = (weight * sdf[corner]).sum(-1)
    rgb = torch.stack([(weight * colors[corner][..., c]).sum(-1) for c in range(3)], -1)
    cdf = torch.where(there, 1.0 / (1.0 + torch.exp(-value * sharp)), torch.zeros_like(value))
    outer = torch.ones_like(cdf[:, 0])
    outer_slope = torch.zeros_like(outer)
    clear = torch.ones_like(outer)
    acc = torch.zeros((which.shape[0], 3), dtype=torch.float64, device=faces.device)
    steps = []
    for l in range(shells):
        on = there[:, l]
        raw = (outer - cdf[:, l] + 1e-5) / (outer + 1e-5)
        alpha = raw.clamp(0.0, 1.0) * on
        acc = acc + rgb[:, l] * (clear * alpha)[:, None]
        slope = cdf[:, l] * (1.0 - cdf[:, l])  # d cdf / d (sdf x sharpness)
        steps.append((on, raw, alpha, clear, acc, outer, outer_slope, slope))
        clear = clear * (1.0 - alpha)
        outer = torch.where(on, cdf[:, l], outer)
        outer_slope = torch.where(on, slope, outer_slope)
    image[which, :3], image[which, 3] = acc, clear
    if dl is None:
        return image, None, None
    d_image = dl(image)[which]
    d_rgb, d_clear = d_image[:, :3], d_image[:, 3]
    grad_rgb = torch.zeros_like(rgb)
    grad_value = torch.zeros_like(value)
    seen = torch.zeros_like(there[:, 0])
    before = torch.zeros_like(which)  # slot of the last hit
    pending = torch.zeros_like(clear)
    pixels = torch.arange(which.shape[0], device=which.device)
    for l, (on, raw, alpha, t, so_far, oc, oc_slope, slope) in enumerate(steps):
        inv = 1.0 / (1.0 - alpha + 1e-6)
        grad_rgb[:, l] = (alpha * t)[:, None] * d_rgb
        d_alpha = (d_rgb * (t[:, None] * rgb[:, l] - (acc - so_far) * inv[:, None])).sum(1) - d_clear * clear * inv
        d_raw = d_alpha * ((raw > 0.0) & (raw < 1.0) & on)
        den = oc + 1e-5
        d_inner = -d_raw / den
        d_outer = d_raw / den - d_raw * (oc - cdf[:, l] + 1e-5) / (den * den)
        close = on & seen  # the hit before this one gets the rest of its gradient
        pending = pending + d_outer * oc_slope * sharp * close
        slot = before if fused else torch.full_like(before, max(l - 1, 0))
        grad_value[pixels[close], slot[close]] += pending[close]
        pending = torch.where(on, d_inner * slope * sharp, pending)
        before = torch.where(on, torch.full_like(before, l), before)
        seen = seen | on
    slot = before if fused else torch.full_like(before, shells - 1)
    grad_value[pixels[seen], slot[seen]] += pending[seen]
    if fused and shells > 1:  # the next hit's weights
        weight[:, :-1] = torch.where(there[:, 1:, None], weight[:, 1:], weight[:, :-1])
    grad_colors, grad_sdf = torch.zeros_like(colors), torch.zeros_like(sdf)
    for l in range(shells):
        on = there[:, l]
        for q in range(3):
            to, w = corner[on, l, q], weight[on, l, q]
            grad_sdf.index_add_(0, to, w * grad_value[on, l])
            grad_colors.index_add_(0, to, w[:, None] * grad_rgb[on, l])
    return image, grad_colors, grad_sdf


def _exact_render(s, kind):
    case = s["case"]
    fused, ssaa = case.get("mode", "fused") == "fused", case.get("ssaa", 1)
    sh, vertices, background = s["vertex_sh"].detach().double(), s["vertices"].double(), s["background"].double()
    grad_sh, grad_sdf = torch.zeros_like(sh), torch.zeros(sh.shape[1], dtype=torch.float64, device=sh.device)
    count = sum(3 * h * w for h, w in s["shapes"])
    images, loss = [], 0.0
    for camera, (h, w) in enumerate(s["shapes"]):
        big_h, big_w = h * ssaa, w * ssaa
        intr = s["intrinsics"][camera] * torch.tensor((ssaa, ssaa, 1.0), device=sh.device)[:, None]
        eye = torch.linalg.inv(s["extrinsics"][camera].double())[:3, 3]
        basis = _basis(torch.nn.functional.normalize(vertices - eye, dim=1, eps=0.0), case["sh_degree"])
        plain = sum(b[:, None] * c for b, c in zip(basis, sh)) + 0.5

        def shown(image):
            blend = image[:, :3] + image[:, 3:] * background
            return blend.reshape(h, ssaa, w, ssaa, 3).mean(dim=(1, 3))

        def slope(image):
            mean = shown(image)
            d = 2.0 * (mean - s["targets"][camera].permute(1, 2, 0).double()) / count
            if fused:  # clipped
                d = d * ((mean >= 0.0) & (mean <= 1.0))
            d = (d / ssaa**2)[:, None, :, None].expand(h, ssaa, w, ssaa, 3).reshape(-1, 3)
            return torch.cat((d, (d * background).sum(1, keepdim=True)), 1)

        raw, grad_colors, d_sdf = _exact_camera(s, camera, big_h, big_w, intr, fused, plain.clamp(min=0.0),
                                                None if kind == "view" else slope)
        image = shown(raw)
        image = (image.clamp(0.0, 1.0) if fused else image).permute(2, 0, 1)
        images.append(image)
        if kind != "view":
            loss = loss + ((image - s["targets"][camera].double()) ** 2).sum() / count
            grad_sdf += d_sdf
            grad_colors = grad_colors * (plain > 0.0)
            for c, b in enumerate(basis):
                grad_sh[c] += b[:, None] * grad_colors
    out = {"images": images if kind == "cameras" else torch.stack(images)}
    return out if kind == "view" else {**out, "loss": loss, "grad_sdf": grad_sdf, "grad_sh": grad_sh}
