"""The work that programs have this package do: workloads, one pass of each, and what 64-bit arithmetic gives.

`listed()` names the workloads, `draw(rng)` gives others of the same ranges, `prepare(case, seed)` makes what a
program has in hand before the call (point clouds on the device, or on the host for the batch call), `run(state)`
is one pass through the public API, `work(case)` the bytes and operations of a pass that its definition asks for,
and `exact(case, seed)` its floating-point results from plain torch in 64 bits.
"""

import math

import torch

import mojo_poissonrecon_b200 as mpr
from mojo_poissonrecon_b200 import batch

DEVICE = "cuda"
TOL = 1e-8


def listed():
    return [
        # The first call in the README: 2,000 points on the unit sphere, a 33^3 grid, five V-cycles.  Launch latency.
        dict(name="recon-2k-d5", kind="recon", shape="sphere", points=2000, depth=5, cycles=5, precision="fp64",
             confidence=False),
        # An ordinary scan with every default of `reconstruct`: FP64, four V-cycles, depth 6.
        dict(name="recon-13k-d6", kind="recon", shape="ellipsoid", points=13337, depth=6, cycles=4, precision="fp64",
             confidence=False),
        # The larger of the two published full reconstructions: 20,000 points at depth 7, default solver.
        dict(name="recon-20k-d7", kind="recon", shape="sphere", points=20000, depth=7, cycles=4, precision="fp64",
             confidence=False),
        # A dense scan with confidence-weighted normals through the default (FP64, fixed cycles) solver.
        dict(name="recon-1m-d8", kind="recon", shape="torus", points=1_000_000, depth=8, cycles=4, precision="fp64",
             confidence=True),
        # The plain FP64 side of the depth-8 comparison: V-cycles to a relative residual of 1e-8, all grids returned.
        dict(name="solve-1m-d8-tol", kind="solve", shape="torus", points=1_000_000, depth=8, precision="fp64",
             confidence=True),
        # A served request of the median size: FP32-refined to 1e-8, mesh out.
        dict(name="refined-50k-d6", kind="recon", shape="ellipsoid", points=50021, depth=6, cycles=4,
             precision="fp32_refined", confidence=False),
        # The headline workload: one million points, depth 8, FP32-refined to 1e-8, mesh out.
        dict(name="refined-1m-d8", kind="recon", shape="torus", points=1_000_000, depth=8, cycles=4,
             precision="fp32_refined", confidence=True),
        # The largest served request: two million points at depth 9; a program that wants the grids themselves.
        dict(name="refined-2m-d9", kind="solve", shape="torus", points=1_999_999, depth=9, precision="fp32_refined",
             confidence=False),
        # Many uneven clouds (1k to 200k points, depths 5 to 8) from host arrays to device meshes in one call.
        dict(name="batch-20", kind="batch", clouds=20, min_points=1000, max_points=200_000, min_depth=5, max_depth=8),
        # Surface extraction alone from a program's own grid, of a side that is no power of two plus one.
        dict(name="extract-230", kind="extract", side=230),
        # The flat octree alone, at the deepest grid depth.
        dict(name="octree-1m-d10", kind="octree", shape="torus", points=1_000_003, depth=10),
        # Colours carried onto a mesh: three channels of a million samples at 160,000 vertices.
        dict(name="attributes-1m-d8", kind="attributes", shape="torus", points=1_000_000, vertices=160_001,
             channels=3, depth=8, confidence=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("recon", "recon", "refined", "refined", "solve", "defect", "batch", "extract", "octree",
                       "attributes"))
    shape = rng.choice(("sphere", "ellipsoid", "torus"))
    confidence = rng.random() < 0.5
    if kind == "recon":
        depth = rng.randint(4, 8)
        return dict(kind=kind, shape=shape, points=_log(rng, 1000, min(1_000_000, 1000 * 4 ** (depth - 3))), depth=depth,
                    cycles=rng.randint(3, 6), precision="fp64", confidence=confidence)
    if kind == "refined":
        depth = rng.randint(5, 9)
        return dict(kind=rng.choice(("recon", "solve")), shape=shape, points=_log(rng, 2000, 400 * 4 ** (depth - 3)),
                    depth=depth, cycles=4, precision="fp32_refined", confidence=confidence)
    if kind in ("solve", "defect"):
        depth = rng.randint(5, 8) if kind == "solve" else rng.randint(5, 7)
        return dict(kind="solve", shape=shape, points=_log(rng, 2000, 1000 * 4 ** (depth - 3)), depth=depth,
                    precision="fp64" if kind == "solve" else "fp32_defect", confidence=confidence)
    if kind == "batch":
        return dict(kind=kind, clouds=rng.randint(5, 20), min_points=1000, max_points=_log(rng, 10_000, 200_000),
                    min_depth=5, max_depth=rng.randint(6, 8))
    if kind == "extract":
        return dict(kind=kind, side=_log(rng, 33, 300))
    if kind == "octree":
        return dict(kind=kind, shape=shape, points=_log(rng, 10_000, 2_000_000), depth=rng.randint(4, 12))
    return dict(kind=kind, shape=shape, points=_log(rng, 10_000, 1_000_000), vertices=_log(rng, 5000, 200_000),
                channels=rng.randint(1, 5), depth=rng.randint(5, 8), confidence=confidence)


# ---- inputs ---------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _rand(g, *size):
    return torch.rand(*size, generator=g, device=DEVICE, dtype=torch.float64)


def _randn(g, *size):
    return torch.randn(*size, generator=g, device=DEVICE, dtype=torch.float64)


def _cloud(shape, count, g, noise=0.0, confidence=False):
    """Area-uniform samples of a surface inside [-1, 1]^3 with outward normals."""
    if shape == "sphere":
        z, theta = 2.0 * _rand(g, count) - 1.0, 2.0 * math.pi * _rand(g, count)
        r = torch.sqrt(1.0 - z * z)
        points = torch.stack((r * torch.cos(theta), r * torch.sin(theta), z), 1)
        normals = points.clone()
    elif shape == "torus":
        major, minor = 0.6, 0.25
        phi = 2.0 * math.pi * _rand(g, 2 * count + 512)
        phi = phi[_rand(g, phi.numel()) < (major + minor * torch.cos(phi)) / (major + minor)][:count]
        theta = 2.0 * math.pi * _rand(g, count)
        ring = major + minor * torch.cos(phi)
        points = torch.stack((ring * torch.cos(theta), ring * torch.sin(theta), minor * torch.sin(phi)), 1)
        normals = torch.stack((torch.cos(phi) * torch.cos(theta), torch.cos(phi) * torch.sin(theta), torch.sin(phi)), 1)
    else:  # ellipsoid with random semi-axes
        axes = 0.2 + 0.7 * _rand(g, 3)
        u = _randn(g, 6 * count + 512, 3)
        u = u / u.norm(dim=1, keepdim=True)
        element = (u * axes.roll(-1) * axes.roll(-2)).norm(dim=1)
        u = u[_rand(g, len(u)) * element.max() < element]
        u = u.repeat(-(-count // len(u)), 1)[:count]
        points, normals = u * axes, u / axes
        normals = normals / normals.norm(dim=1, keepdim=True)
    if noise:
        points = points + noise * _randn(g, count, 3)
    if confidence:
        normals = normals * (0.5 + _rand(g, count, 1))
    return points.contiguous(), normals.contiguous()


def _unit(points):
    """Into the unit cube with a margin, as `reconstruct` does by itself."""
    lo, hi = points.amin(0), points.amax(0)
    width = 1.1 * (hi - lo).max()
    return ((points - (0.5 * (lo + hi) - 0.5 * width)) / width).contiguous()


def _waves(side, g):
    """A smooth scalar grid whose zero surface fills the cube: a few plane waves of random phase."""
    t = torch.linspace(0.0, 1.0, side, dtype=torch.float64, device=DEVICE)
    field = torch.zeros(side, side, side, dtype=torch.float64, device=DEVICE)
    for axis_freq in ((3.0, 2.0, 1.0), (1.0, 3.0, 2.0), (2.0, 1.0, 3.0)):
        phase = 2.0 * math.pi * _rand(g, 1)
        k = [2.0 * math.pi * f for f in axis_freq]
        field += torch.sin(k[0] * t[:, None, None] + k[1] * t[None, :, None] + k[2] * t[None, None, :] + phase)
    return field


def _mesh_buffers(side):
    """Buffers of a fixed size that a program keeps for the meshes it is given: vertices, faces, vertex densities.
    The surfaces here cross fewer than 24 side^2 cells."""
    rows = 24 * side * side
    return (torch.zeros(rows, 3, dtype=torch.float64, device=DEVICE),
            torch.zeros(2 * rows, 3, dtype=torch.int64, device=DEVICE),
            torch.zeros(rows, dtype=torch.float64, device=DEVICE))


def _tree_buffers(points, depth):
    nodes = sum(min(8 ** level, points) for level in range(depth + 1))
    return [torch.zeros(rows, dtype=torch.int64, device=DEVICE) for rows in [nodes] * 5 + [points]]


def _fill(buffers, arrays):
    """The arrays at the start of the program's buffers, and how many rows they have."""
    for buffer, array in zip(buffers, arrays):
        buffer[:len(array)] = array
    return [*buffers, *(len(array) for array in arrays)]


def _mesh_out(buffers, mesh):
    return _fill(buffers, (mesh.vertices, mesh.faces, mesh.density))


def _tree_out(buffers, tree):
    return _fill(buffers, (tree.depth, tree.morton, tree.parent, tree.child_start, tree.child_count, tree.point_leaf))


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    state = dict(case=case)
    if kind in ("recon", "extract"):
        state["mesh"] = _mesh_buffers(case["side"] if kind == "extract" else 2 ** case["depth"] + 1)
    if kind in ("solve", "octree"):
        state["tree"] = _tree_buffers(case["points"], case["depth"])
    if kind in ("recon", "solve"):
        points, normals = _cloud(case["shape"], case["points"], g, 0.002, case["confidence"])
        state["points"], state["normals"] = (points if kind == "recon" else _unit(points)), normals
    elif kind == "octree":
        state["points"] = _unit(_cloud(case["shape"], case["points"], g, 0.002)[0])
    elif kind == "extract":
        state["field"] = _waves(case["side"], g)
        state["density"] = 1.0 + _waves(case["side"], g).abs()
    elif kind == "attributes":
        state["points"], state["normals"] = _cloud(case["shape"], case["points"], g, 0.0, case["confidence"])
        state["values"] = _rand(g, case["points"], case["channels"])
        state["vertices"] = _cloud("torus" if case["shape"] == "torus" else "sphere", case["vertices"], g)[0] * 0.99
    else:  # batch: host arrays
        clouds = []
        size = _rand(g, case["clouds"]).tolist()
        spread = math.log(case["max_points"] / case["min_points"])
        for k in range(case["clouds"]):
            d = case["max_depth"] - k % (case["max_depth"] - case["min_depth"] + 1)
            count = int(case["min_points"] * math.exp(spread * (k + size[k]) / case["clouds"]))
            points, normals = _cloud(("ellipsoid", "torus")[k % 2], count, g)
            clouds.append((points.cpu().numpy(), normals.cpu().numpy(), d))
        state["clouds"] = clouds
        state["mesh"] = _mesh_buffers(math.isqrt(sum((2 ** d + 1) ** 2 for _, _, d in clouds)) + 1)
    return state


# ---- one pass ---------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "recon":
        fp64 = case["precision"] == "fp64"
        mesh = mpr.reconstruct(state["points"], state["normals"], depth=case["depth"], cycles=case["cycles"],
                               confidence=case["confidence"], precision=case["precision"], tol=None if fp64 else TOL,
                               device_out=True)
        out = dict(mesh=_mesh_out(state["mesh"], mesh), iso=mesh.iso_value)
        if fp64:  # a fixed number of cycles: its residual is a result; elsewhere it says that TOL was met
            out["residual_norm"] = mesh.residual_norm
        return out
    if kind == "solve":
        sol = mpr.solve_screened_poisson(state["points"], state["normals"], depth=case["depth"],
                                         confidence=case["confidence"], precision=case["precision"], tol=TOL,
                                         device_out=True)
        return dict(field=sol.field, density=sol.density, screen=sol.screen, rhs=sol.rhs, iso=sol.iso_value,
                    octree=_tree_out(state["tree"], sol.octree))
    if kind == "octree":
        return _tree_out(state["tree"], mpr.build_octree(state["points"], case["depth"], device_out=True))
    if kind == "extract":
        return _mesh_out(state["mesh"], mpr.extract_isosurface(state["field"], iso_value=0.0,
                                                               density=state["density"], device_out=True))
    if kind == "attributes":
        return mpr.interpolate_attributes(state["points"], state["normals"], state["values"], state["vertices"],
                                          depth=case["depth"], confidence=case["confidence"], device_out=True)
    # one buffer of each kind for the whole batch, the meshes one after another
    meshes = batch.reconstruct_many(state["clouds"], tol=TOL, device_out=True)
    parts = [torch.cat([getattr(m, name) for m in meshes]) for name in ("vertices", "faces", "density")]
    return dict(mesh=_fill(state["mesh"], parts), counts=[len(m.faces) for m in meshes],
                iso=torch.tensor([m.iso_value for m in meshes], dtype=torch.float64))


# ---- what a pass cannot do without --------------------------------------------------

def _solve_work(points, depth, cycles):
    """Points in, the grids out, and per cycle the iterate read and written and its two coefficient grids read
    once on every level; per node and cycle six sweeps' and a residual's additions."""
    nodes = (2 ** depth + 1) ** 3
    return points * 48 + nodes * 32 + cycles * nodes * 32 * 8 / 7, cycles * nodes * 96 * 8 / 7 + points * 200


def work(case):
    kind = case["kind"]
    cycles = {"fp64": 31, "fp32_refined": 6, "fp32_defect": 7}  # measured to TOL on these surfaces
    if kind in ("recon", "solve"):
        fixed = kind == "recon" and case["precision"] == "fp64"
        b, f = _solve_work(case["points"], case["depth"], case["cycles"] if fixed else cycles[case["precision"]])
        return dict(bytes=b, flops=f)
    if kind == "batch":
        middle = math.sqrt(case["min_points"] * case["max_points"])
        got = [_solve_work(middle, d, cycles["fp32_refined"]) for d in range(case["min_depth"], case["max_depth"] + 1)]
        return dict(bytes=case["clouds"] * sum(b for b, _ in got) / len(got),
                    flops=case["clouds"] * sum(f for _, f in got) / len(got))
    if kind == "octree":
        return dict(bytes=case["points"] * (24 + 8 + 4 * 40 // 3), flops=case["points"] * case["depth"] * 12)
    if kind == "extract":
        # both grids' values at the surface's cells, the field once, the mesh out (about 10 side^2 cells cross it)
        return dict(bytes=case["side"] ** 3 * 8 + case["side"] ** 2 * 10 * (64 + 32 + 48),
                    flops=case["side"] ** 3 + case["side"] ** 2 * 1000)
    c = case["channels"]
    return dict(bytes=case["points"] * (48 + 8 * c) + case["vertices"] * (24 + 8 * c),
                flops=(case["points"] + case["vertices"]) * 8 * 3 * (c + 2))


# ---- the same results in 64 bits by plain torch ---------------------------------------

def _cells(unit, res):
    g = unit * res
    i = g.long().clamp(0, res - 1)
    return i, (g - i).clamp(0.0, 1.0)


def _corners(unit, n):
    """(node index, trilinear weight) of each point's eight corners."""
    i, f = _cells(unit, n - 1)
    for c in range(8):
        d = torch.tensor([c & 1, (c >> 1) & 1, c >> 2], device=unit.device)
        w = torch.where(d == 1, f, 1.0 - f).prod(1)
        at = i + d
        yield (at[:, 2] * n + at[:, 1]) * n + at[:, 0], w


def _interpolate(grid, unit):
    flat, n = grid.reshape(-1), grid.shape[0]
    return sum(flat[at] * w for at, w in _corners(unit, n))


def _splat(unit, normals, depth, confidence, spn=1.5):
    n = 2 ** depth + 1
    res, zero = n - 1, lambda: torch.zeros(n ** 3, dtype=torch.float64, device=unit.device)
    length = normals.norm(dim=1)
    weight = length if confidence else torch.ones_like(length)
    screen = zero()
    for at, w in _corners(unit, n):
        screen.index_add_(0, at, w * weight)
    density = 2.0 * screen
    factor = (_interpolate(density.view(n, n, n), unit) / spn).clamp(min=1.0)
    vectors = []
    for a in range(3):
        v = zero()
        for at, w in _corners(unit, n):
            v.index_add_(0, at, -(normals[:, a] / length) * w * weight * res / factor)
        vectors.append(v.view(n, n, n))
    screen = screen.view(n, n, n)
    rhs = 4.0 * screen * (res * res) * 0.5
    for v, axis in zip(vectors, (2, 1, 0)):
        rhs -= torch.gradient(v, spacing=1.0 / res, dim=axis)[0]
    return density.view(n, n, n) / spn, screen, rhs


class _Level:
    def __init__(self, screen):
        n = screen.shape[0]
        end = torch.full((n,), 2.0, dtype=torch.float64, device=screen.device)
        end[0] = end[-1] = 1.0
        self.h2 = float(n - 1) ** 2
        self.diagonal = (end[:, None, None] + end[None, :, None] + end[None, None, :] + 4.0 * screen) * self.h2
        odd = torch.arange(n, device=screen.device) & 1
        self.colour = (odd[:, None, None] ^ odd[None, :, None] ^ odd[None, None, :]).bool()
        self.n = n

    def neighbours(self, v):
        s = torch.zeros_like(v)
        for axis in range(3):
            s.narrow(axis, 1, self.n - 1).add_(v.narrow(axis, 0, self.n - 1))
            s.narrow(axis, 0, self.n - 1).add_(v.narrow(axis, 1, self.n - 1))
        return s

    def relax(self, v, rhs, sweeps):
        for _ in range(sweeps):
            for c in (False, True):
                new = self.neighbours(v).mul_(self.h2).add_(rhs).div_(self.diagonal)
                v = torch.where(self.colour == c, new, v)
        return v

    def apply(self, v):
        return self.diagonal * v - self.h2 * self.neighbours(v)


def _restrict(v):
    """Full weighting, renormalised at the boundary, one axis at a time."""
    for axis in range(3):
        v = v.movedim(axis, 0)
        out = 2.0 * v[::2]
        out[1:] += v[1::2]
        out[:-1] += v[1::2]
        out[1:-1] /= 4.0
        out[0] /= 3.0
        out[-1] /= 3.0
        v = out.movedim(0, axis)
    return v.contiguous()


def _prolong(v):
    for axis in range(3):
        v = v.movedim(axis, 0)
        out = v.new_empty((2 * v.shape[0] - 1, *v.shape[1:]))
        out[::2] = v
        out[1::2] = 0.5 * (v[1:] + v[:-1])
        v = out.movedim(0, axis)
    return v


def _levels(screen):
    levels = [_Level(screen)]
    while screen.shape[0] > 3:
        screen = 4.0 * _restrict(screen)
        levels.append(_Level(screen))
    return levels


def _v_cycle(levels, v, rhs, k=0):
    level = levels[k]
    if level.n <= 3:
        return level.relax(v, rhs, 40)
    v = level.relax(v, rhs, 3)
    coarse = _restrict(rhs - level.apply(v))
    v = v + _prolong(_v_cycle(levels, torch.zeros_like(coarse), coarse, k + 1))
    return level.relax(v, rhs, 3)


def _converged(levels, rhs, iterations=60):
    """Flexible conjugate gradients with that V-cycle to the last digits that 64 bits hold."""
    x = torch.full_like(rhs, 0.5)
    goal, p, ap = 1e-13 * rhs.norm(), None, None
    for _ in range(iterations):
        r = rhs - levels[0].apply(x)
        if r.norm() <= goal:
            break
        z = _v_cycle(levels, torch.zeros_like(r), r)
        p = z if p is None else z - ((z * ap).sum() / (p * ap).sum()) * p
        ap = levels[0].apply(p)
        x = x + ((p * r).sum() / (p * ap).sum()) * p
    return x


def _surface(field, density, iso):
    """Dual-contouring vertices (unit cube) and their densities, cells in z, y, x order."""
    m = field.shape[0] - 1
    corner = lambda grid, c: grid[c >> 2:(c >> 2) + m, (c >> 1) & 1:((c >> 1) & 1) + m, c & 1:(c & 1) + m]
    below = sum((corner(field, c) < iso).to(torch.int8) for c in range(8))
    at = ((below > 0) & (below < 8)).nonzero()
    value = [corner(field, c)[tuple(at.T)] for c in range(8)]
    total, roots = torch.zeros(len(at), 3, dtype=torch.float64, device=field.device), 0
    for axis in range(3):
        for c in range(8):
            if c >> axis & 1:
                continue
            v0, v1 = value[c], value[c | 1 << axis]
            cross = (v0 < iso) != (v1 < iso)
            t = torch.where(cross, (iso - v0) / (v1 - v0), 0.0).clamp(0.0, 1.0)
            for a in range(3):
                total[:, a] += torch.where(cross, t if a == axis else float(c >> a & 1), 0.0)
            roots = roots + cross
    vertices = (at.flip(1) + total / roots[:, None]) / m
    return vertices, sum(corner(density, c)[tuple(at.T)] for c in range(8)) / 8.0


def _surface_out(state, vertices, density):
    """As _mesh_out lays a mesh out, without its whole numbers."""
    return [_fill(state["mesh"][:1], (vertices,))[0], None, _fill(state["mesh"][2:], (density,))[0]]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("octree", "batch"):  # whole numbers; a mesh whose topology hangs on the iteration's last digits
        return None
    s = prepare(case, seed)
    if kind == "extract":
        return _surface_out(s, *_surface(s["field"], s["density"], 0.0))
    if kind == "attributes":
        lo, hi = s["points"].amin(0), s["points"].amax(0)
        width = 1.1 * (hi - lo).max()
        origin = 0.5 * (lo + hi) - 0.5 * width
        unit, at_vertices = (s["points"] - origin) / width, (s["vertices"] - origin) / width
        n = 2 ** case["depth"] + 1
        weight = s["normals"].norm(dim=1) if case["confidence"] else torch.ones_like(unit[:, 0])
        sums = []
        for c in range(case["channels"] + 1):
            grid = torch.zeros(n ** 3, dtype=torch.float64, device=unit.device)
            for at, w in _corners(unit, n):
                grid.index_add_(0, at, w * weight * (s["values"][:, c] if c < case["channels"] else 1.0))
            sums.append(_interpolate(grid.view(n, n, n), at_vertices))
        total = sums.pop()
        return torch.stack([torch.where(total > 0, v / total, 0.0) for v in sums], 1)
    points, normals = s["points"], s["normals"]
    if kind == "recon":
        lo, hi = points.amin(0), points.amax(0)
        width = 1.1 * (hi - lo).max()
        origin = 0.5 * (lo + hi) - 0.5 * width
        points = (points - origin) / width
    density, screen, rhs = _splat(points, normals, case["depth"], case["confidence"])
    levels = _levels(screen)
    fixed = kind == "recon" and case["precision"] == "fp64"
    if fixed:
        field = torch.full_like(rhs, 0.5)
        for _ in range(case["cycles"]):
            field = _v_cycle(levels, field, rhs)
    else:
        field = _converged(levels, rhs)
    weight = normals.norm(dim=1) if case["confidence"] else torch.ones_like(normals[:, 0])
    iso = float((_interpolate(field, points) * weight).sum() / weight.sum())
    if kind == "solve":
        return dict(field=field, density=density, screen=screen, rhs=rhs, iso=iso, octree=None)
    if not fixed:  # the mesh's topology hangs on the iteration's last digits
        return dict(mesh=None, iso=iso)
    vertices, values = _surface(field, density, iso)
    return dict(mesh=_surface_out(s, vertices * width + origin, values), iso=iso,
                residual_norm=float((rhs - levels[0].apply(field)).norm()))
