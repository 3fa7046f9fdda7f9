"""The calls that a frame of the fusion pipeline is made of, each with inputs
of its own, at the sizes this repository's workloads, tests and benchmark use.

The scenes are synthetic and are made on the GPU from the seed: a bumpy
surface about 1.1 m in front of a pinhole camera (one point or vertex per
pixel, deformation nodes on a jittered pixel lattice) and spheres with evenly
spread nodes, both with a smooth node warp, sensor noise of 1 mm and a few
invalid or outlying samples.

    listed()           the cases that are measured
    draw(rng)          one more case of the same ranges
    prepare(case, s)   inputs and handles on the GPU, from the seed alone
    run(state)         one pass through the public entry points
    work(case)         the bytes and operations a pass cannot do without
    exact(case, s)     the pass's results in 64 bits, in plain torch
"""
import math

import numpy as np
import torch

from cudafusion_b200 import _lib
from cudafusion_b200 import learned
from cudafusion_b200.corr import CorrParams, CorrespondenceSearch, DeviceCorrFrame
from cudafusion_b200.linesearch import LineSearch, LineSearchParams
from cudafusion_b200.raster import DeviceMesh, LiveSurfaceRaster, voxel_grid
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params
from cudafusion_b200.tsdf import TSDFVolume, TsdfParams

DEV = "cuda"
F64 = torch.float64
CLAMPS = (0.12, 0.04)  # the pipeline's twist clamps (rad, m)
VOLUME = 1.536  # metres along x that a volume spans (256 voxels of 6 mm)
ORIGIN = (-0.768, -0.768, 0.5)


def listed():
    return [
        # The small plain solve: a sphere of 256 nodes, 20k correspondences.
        # Latency, not bytes, is what a user waits for here.
        dict(name="solve sphere 256", kind="solve", scene="sphere", nodes=256, corrs=20000, gn=5, pcg=10),
        # The per-frame solve at the headline size: a 640x480 depth frame,
        # 2048 nodes, warm-started from the previous frame.
        dict(name="solve frame 2048", kind="solve", scene="frame", nodes=2048, width=640, height=480, gn=5, pcg=20),
        # The largest single problem a warp field holds: 8192 nodes and a
        # 1280x960 depth frame.
        dict(name="solve frame 8192", kind="solve", scene="frame", nodes=8192, width=1280, height=960, gn=5, pcg=20),
        # The reference solver's own call: one linearisation on the records of
        # a correspondence search, of which a part is invalid.
        dict(name="linearize frame", kind="linearize", nodes=2000, width=640, height=480, pcg=10, invalid=0.12),
        # Many uneven problems in one call: training data, offline runs.
        dict(name="batch 64", kind="batch", problems=64, low=500, high=8000, per_node=150, gn=5, pcg=20),
        # The learned start: features, network, gate and one GN iteration.
        dict(name="learned frame", kind="learned", nodes=2048, width=640, height=480),
        # The network's training direction: loss and gradients of a batch of
        # eight frames' graphs.
        dict(name="network gradients", kind="gradients", nodes=2048, frames=8),
        # The projective search of a frame at the stock thresholds.
        dict(name="search 640x480 r50", kind="search", width=640, height=480, radius=50, dist=0.2, angle=0.0,
             voxels=True),
        # Skinning and rasterising a frame's mesh into the live maps.
        dict(name="predict 153k triangles", kind="predict", width=640, height=480, stride=2, nodes=2048, dims=256),
        # A GN step's line search: ten predictions and searches.
        dict(name="line search 320x240", kind="linesearch", width=320, height=240, stride=1, nodes=1024, dims=128,
             radius=20),
        # A frame fused into the canonical volume: warped, gated by the counts.
        dict(name="integrate 256^3", kind="integrate", width=640, height=480, dims=256, nodes=1728, warp=True),
        # The volume's node lists, renewed after each change of the graph.
        dict(name="voxel lists 256^3", kind="voxelknn", width=640, height=480, dims=256, nodes=1728),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "linearize", "batch", "learned", "gradients", "search", "search", "predict",
                       "linesearch", "integrate", "voxelknn"])
    if kind in ("solve", "linearize", "learned"):
        w = _log(rng, 96, 1100)
        c = dict(kind=kind, nodes=_log(rng, 64, 6000), width=w, height=max(64, int(w * rng.uniform(0.6, 0.8))))
        c["nodes"] = min(c["nodes"], c["width"] * c["height"] // 40)
        if kind == "linearize":
            c.update(pcg=rng.randint(5, 20), invalid=round(rng.uniform(0.0, 0.4), 3))
        elif kind == "solve":
            c.update(scene="frame", gn=rng.randint(1, 6), pcg=rng.randint(5, 20))
            if rng.random() < 0.4:
                n = _log(rng, 100, 3000)
                c = dict(kind=kind, scene="sphere", nodes=n, corrs=int(n * rng.uniform(60, 180)), gn=c["gn"],
                         pcg=c["pcg"])
        return c
    if kind == "batch":
        low = _log(rng, 100, 1500)
        return dict(kind=kind, problems=rng.randint(2, 40), low=low, high=low * rng.randint(2, 4),
                    per_node=rng.randint(80, 180), gn=rng.randint(2, 6), pcg=rng.randint(8, 20))
    if kind == "gradients":
        return dict(kind=kind, nodes=_log(rng, 100, 4000), frames=rng.randint(1, 8))
    w = _log(rng, 80, 640)
    h = max(48, int(w * rng.uniform(0.6, 0.8)))
    if kind == "search":
        return dict(kind=kind, width=w, height=h, radius=_log(rng, 1, 50), dist=rng.choice([0.02, 0.05, 0.2]),
                    angle=rng.choice([0.0, 0.0, 0.5]), voxels=rng.random() < 0.5)
    dims = rng.randint(64, 256)
    if kind == "integrate":
        return dict(kind=kind, width=w, height=h, dims=dims, nodes=_log(rng, 64, 3000), warp=rng.random() < 0.8)
    if kind == "voxelknn":
        return dict(kind=kind, width=w, height=h, dims=dims, nodes=_log(rng, 64, 6000))
    c = dict(kind=kind, width=w, height=h, stride=rng.randint(1, 3), nodes=_log(rng, 64, 3000), dims=dims)
    if kind == "linesearch":
        c["radius"] = rng.randint(2, 24)
    c["nodes"] = min(c["nodes"], w * h // 40)
    return c


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], -1)


def _qconj(q):
    return torch.cat([-q[..., :3], q[..., 3:]], -1)


def _qrot(q, v):
    return _qmul(_qmul(q, torch.cat([v, torch.zeros_like(v[..., :1])], -1)), _qconj(q))[..., :3]


def _qexp(w):
    th = w.norm(dim=-1, keepdim=True)
    s = torch.where(th > 1e-9, torch.sin(0.5 * th) / th.clamp_min(1e-30), torch.full_like(th, 0.5))
    return torch.cat([w * s, torch.cos(0.5 * th)], -1)


def _dq(q, t):
    """[N, 8]: a rotation and a node-centred translation as a dual quaternion."""
    return torch.cat([q, 0.5 * _qmul(torch.cat([t, torch.zeros_like(t[:, :1])], -1), q)], -1)


def _smooth(g, x, amplitude, scale):
    """A low-frequency vector field over the points x, at most `amplitude` long."""
    f = torch.zeros_like(x)
    for _ in range(3):
        f += torch.sin(x @ (_randn(g, 3) / scale) + 2 * math.pi * _rand(g, 1))[:, None] * _randn(g, 3)
    return f * (amplitude / f.norm(dim=-1).max().clamp_min(1e-12))


def _warp(g, pos, rot, trans, scale):
    return _dq(_qexp(_smooth(g, pos, rot, scale)), _smooth(g, pos, trans, scale))


def _skin(p, ids, ws, pos, T):
    """Points blended by their nodes' dual quaternions, and the blended rotations."""
    q, d = T[:, :4], T[:, 4:]
    n = q.norm(dim=-1, keepdim=True)
    t = 2 * _qmul(d, _qconj(q))[:, :3] + pos - _qrot(q, pos)
    q = q / n
    d = 0.5 * _qmul(torch.cat([t, torch.zeros_like(t[:, :1])], -1), q)
    br, bd = torch.zeros(len(p), 4, device=DEV, dtype=F64), torch.zeros(len(p), 4, device=DEV, dtype=F64)
    total = torch.zeros(len(p), 1, device=DEV, dtype=F64)
    for k in range(4):
        w = torch.where((ids[:, k] >= 0) & (ws[:, k] >= 1e-8), ws[:, k], torch.zeros_like(ws[:, k]))[:, None]
        i = ids[:, k].clamp_min(0)
        s = torch.where((q[i] * br).sum(-1, keepdim=True) < 0, -w, w)
        br = br + s * q[i]
        bd = bd + s * d[i]
        total = total + w
    n = br.norm(dim=-1, keepdim=True).clamp_min(1e-30)
    br, bd = br / n, bd / n
    out = _qrot(br, p) + 2 * _qmul(bd, _qconj(br))[:, :3]
    return torch.where(total < 1e-8, p, out), br


def _weights(d2, radius):
    w = torch.exp(-d2 / (2 * radius * radius))
    s = w.sum(-1, keepdim=True)
    return torch.where(s > 1e-8, w / s.clamp_min(1e-300), torch.zeros_like(w))


def _graph(pos):
    """Each node's 8 nearest, their distances, and the median nearest spacing."""
    k = min(9, len(pos))
    d, i = [], []
    for c in pos.float().split(2048):
        a, b = torch.cdist(c, pos.float(), compute_mode="donot_use_mm_for_euclid_dist").topk(k, largest=False)
        d.append(a[:, 1:])
        i.append(b[:, 1:])
    d, i = torch.cat(d).double(), torch.cat(i)
    return i, d, float(d[:, 0].median())


def _near(points, cand, pos, radius, most=1 << 19):
    """The 4 nearest of each point's candidate nodes (-1: none) and their weights."""
    ids, ws = [], []
    for p, c in zip(points.split(most), cand.split(most)):
        d = ((pos[c.clamp_min(0)] - p[:, None]) ** 2).sum(-1)
        d = torch.where(c < 0, torch.full_like(d, math.inf), d)
        d, o = d.topk(4, largest=False)
        i = torch.where(d < math.inf, c.gather(1, o), torch.full_like(o, -1))
        ids.append(i)
        ws.append(_weights(d, radius))
    return torch.cat(ids), torch.cat(ws)


class Surface:
    """The bumpy surface seen by a width x height camera, with nodes on a
    jittered lattice of its pixels."""

    def __init__(self, g, width, height, nodes):
        W, H = self.W, self.H = width, height
        self.f, self.cx, self.cy = 570.342 * W / 640.0, W / 2.0, H / 2.0
        self.cam = _lib.Camera(self.f, self.f, self.cx, self.cy, W, H)
        self.phase = _rand(g, 2) * 2 * math.pi
        v, u = torch.meshgrid(torch.arange(H, device=DEV, dtype=F64), torch.arange(W, device=DEV, dtype=F64),
                              indexing="ij")
        self.u, self.v = u, v
        self.z = self.depth_at(u, v)
        self.points = self.unproject(self.z).reshape(-1, 3)
        # a lattice somewhat denser than asked for, thinned to the number of nodes
        s = math.sqrt(W * H / (1.06 * nodes))
        nx, ny = max(2, int(W / s)), max(2, int(H / s))
        while nx * ny < nodes:
            nx, ny = nx + 1, ny + 1
        sx, sy = W / nx, H / ny
        jy, jx = torch.meshgrid(torch.arange(ny, device=DEV), torch.arange(nx, device=DEV), indexing="ij")
        un = (jx + 0.5 + 0.5 * (_rand(g, ny, nx) - 0.5)) * sx
        vn = (jy + 0.5 + 0.5 * (_rand(g, ny, nx) - 0.5)) * sy
        keep = torch.sort(torch.randperm(nx * ny, generator=g, device=DEV)[:nodes])[0]
        lattice = torch.full((nx * ny,), -1, device=DEV, dtype=torch.int64)
        lattice[keep] = torch.arange(nodes, device=DEV)
        self.lattice, self.nx, self.ny, self.sx, self.sy = lattice.view(ny, nx), nx, ny, sx, sy
        un, vn = un.reshape(-1)[keep], vn.reshape(-1)[keep]
        zn = self.depth_at(un, vn)
        self.pos = torch.stack([zn * (un - self.cx) / self.f, zn * (vn - self.cy) / self.f, zn], -1)
        self.pos = self.pos.float().double()
        self.nb, self.nd, spacing = _graph(self.pos)
        self.radius = float(np.float32(1.3 * spacing))

    def depth_at(self, u, v):
        return (1.1 + 0.12 * torch.sin(2 * math.pi * 1.5 * u / self.W + self.phase[0])
                * torch.cos(2 * math.pi * v / self.H + self.phase[1]) + 0.06 * u / self.W)

    def unproject(self, z):
        return torch.stack([z * (self.u - self.cx) / self.f, z * (self.v - self.cy) / self.f, z], -1)

    def candidates(self, u, v):
        """The nodes of the 5 x 5 lattice cells around pixels (u, v)."""
        cx, cy = (u / self.sx).long().clamp(0, self.nx - 1), (v / self.sy).long().clamp(0, self.ny - 1)
        out = []
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                x, y = cx + dx, cy + dy
                ok = (x >= 0) & (x < self.nx) & (y >= 0) & (y < self.ny)
                i = self.lattice[y.clamp(0, self.ny - 1), x.clamp(0, self.nx - 1)]
                out.append(torch.where(ok, i, torch.full_like(i, -1)))
        return torch.stack(out, -1)

    def skin_lists(self):
        return _near(self.points, self.candidates(self.u.reshape(-1), self.v.reshape(-1)), self.pos, self.radius)

    def nodes(self):
        return _nodes(self.pos, self.nb, self.nd, self.radius)


def _normals(P):
    """Forward-difference normals of a point map, facing the camera; 0 on the last row and column."""
    n = torch.zeros_like(P)
    a = torch.linalg.cross(P[:-1, 1:] - P[:-1, :-1], P[1:, :-1] - P[:-1, :-1])
    n[:-1, :-1] = -a / a.norm(dim=-1, keepdim=True).clamp_min(1e-30)
    return n


def _nodes(pos, nb, nd, radius):
    """The 96-byte node records as bytes."""
    n, k = nb.shape
    f = torch.zeros(n, 24, device=DEV)
    i = f.view(torch.int32)
    f[:, :3] = pos.float()
    f[:, 5] = -1.0
    f[:, 6] = radius
    i[:, 7:15] = -1
    i[:, 7:7 + k] = nb.int()
    f[:, 15:15 + k] = torch.exp(-nd ** 2 / (2 * radius * radius)).float()
    i[:, 23] = k
    return f.view(torch.uint8).reshape(-1)


def _records(src, dst, nrm, ids, ws, weight, valid):
    """The 76-byte correspondence records as bytes."""
    f = torch.zeros(len(src), 19, device=DEV)
    i = f.view(torch.int32)
    f[:, 0:3], f[:, 3:6], f[:, 6:9] = src.float(), dst.float(), nrm.float()
    i[:, 9:13] = ids.int()
    f[:, 13:17] = ws.float()
    f[:, 17] = weight.float()
    i[:, 18] = valid.int()
    return f.view(torch.uint8).reshape(-1)


def _problem(nodes, canon, corrs, T0):
    p = DeviceProblem.__new__(DeviceProblem)
    p.num_nodes, p.num_corrs = nodes.numel() // 96, corrs.numel() // 76
    p.nodes, p.canon, p.corrs = nodes, canon.float().contiguous(), corrs
    p.init_transforms = T0.float().contiguous().view(torch.uint8).reshape(-1)
    return p


def _frame_problem(g, width, height, nodes, invalid=0.0, past=0):
    """A depth frame's problem; with `past`, the warps of that many frames before too."""
    s = Surface(g, width, height, nodes)
    ids, ws = s.skin_lists()
    rot, trans = _smooth(g, s.pos, math.radians(4.0), 0.5), _smooth(g, s.pos, 0.012, 0.5)

    def at(a):
        return _dq(_qexp(rot * a), trans * a)

    live, q = _skin(s.points, ids, ws, s.pos, at(1.0))
    nrm = _qrot(q, _normals(s.points.view(height, width, 3)).reshape(-1, 3))
    dst = live * (1 + 0.001 * _randn(g, len(live), 1) / live[:, 2:])
    inner = (s.u < width - 1) & (s.v < height - 1)
    if past or not invalid:
        # the canonical points a frame sees
        sel = inner.reshape(-1)
        ids, ws, live, nrm, dst, canon = ids[sel], ws[sel], live[sel], nrm[sel], dst[sel], s.points[sel]
        valid = torch.ones(len(canon), device=DEV, dtype=torch.bool)
        weight = torch.ones(len(canon), device=DEV)
    else:
        # a search's records, one per pixel, those without a match zeroed
        canon = s.points
        valid = inner.reshape(-1) & (_rand(g, len(canon)) >= invalid)
        weight = (0.2 + 0.8 * _rand(g, len(canon))) * valid
        ids = torch.where(valid[:, None], ids, torch.full_like(ids, -1))
        ws, nrm, dst = ws * valid[:, None], nrm * valid[:, None], dst * valid[:, None]
    # the previous frame's warp, four fifths of the way
    warm = at(0.8)
    src = canon
    if invalid:
        src = _skin(canon, ids, ws, s.pos, warm.float().double())[0] * valid[:, None]
    p = _problem(s.nodes(), canon, _records(src, dst, nrm, ids, ws, weight, valid), warm)
    if past:
        p.history = torch.cat([at(0.8 - 0.2 * (k + 1)).float() for k in range(past)]).view(torch.uint8).reshape(-1)
    return p


def _sphere_problem(g, nodes, corrs, max_rot=15.0, max_trans=0.02):
    """Evenly spread nodes on a sphere of 0.3 m about (0, 0, 1), points near
    random nodes, 5 % outliers within 5 cm, an identity start."""
    c = torch.tensor([0.0, 0.0, 1.0], device=DEV, dtype=F64)
    i = torch.arange(nodes, device=DEV, dtype=F64) + 0.5
    phi, th = torch.acos(1 - 2 * i / nodes), math.pi * (1 + 5 ** 0.5) * i
    n = torch.stack([torch.cos(th) * torch.sin(phi), torch.sin(th) * torch.sin(phi), torch.cos(phi)], -1)
    gap = math.sqrt(4 * math.pi / nodes)
    q = _randn(g, 4)
    n = _qrot((q / q.norm()).expand(nodes, 4), n) + 0.15 * gap * _randn(g, nodes, 3)
    n = n / n.norm(dim=-1, keepdim=True)
    pos = (c + 0.3 * n).float().double()
    nb, nd, _ = _graph(pos)
    radius = float(np.float32(0.3 * gap))
    cand = torch.cat([torch.arange(nodes, device=DEV)[:, None], nb, nb[nb[:, :4]].reshape(nodes, -1)], 1)
    cand, order = cand.sort(1)
    cand[:, 1:] = torch.where(cand[:, 1:] == cand[:, :-1], torch.full_like(cand[:, 1:], -1), cand[:, 1:])
    at = torch.randint(nodes, (corrs,), generator=g, device=DEV)
    m = n[at] + gap * (_rand(g, corrs, 3) - 0.5)
    m = m / m.norm(dim=-1, keepdim=True)
    canon = c + 0.3 * m
    ids, ws = [], []
    for a, p in zip(at.split(1 << 19), canon.split(1 << 19)):
        x, y = _near(p, cand[a], pos, radius)
        ids.append(x)
        ws.append(y)
    ids, ws = torch.cat(ids), torch.cat(ws)
    T = _warp(g, pos - c, math.radians(max_rot), max_trans, 0.3)
    live, q = _skin(canon, ids, ws, pos, T)
    nrm = _qrot(q, m)
    dst = live + 0.001 * _randn(g, corrs, 1) * nrm
    out = _rand(g, corrs, 1) < 0.05
    u = _randn(g, corrs, 3)
    dst = torch.where(out, dst + 0.05 * _rand(g, corrs, 1) ** (1 / 3) * u / u.norm(dim=-1, keepdim=True), dst)
    one = torch.ones(corrs, device=DEV)
    ident = torch.zeros(nodes, 8, device=DEV)
    ident[:, 3] = 1.0
    return _problem(_nodes(pos, nb, nd, radius), canon, _records(canon, dst, nrm, ids, ws, one, one > 0), ident)


def _batch_sizes(case):
    """The problems' (nodes, correspondences): the same for every seed."""
    r = np.random.default_rng(case["problems"] * 1000 + case["low"])
    n = r.integers(case["low"], case["high"] + 1, case["problems"])
    return [(int(k), int(k * case["per_node"] * r.uniform(0.8, 1.2))) for k in n]


class Volume:
    """A canonical volume of dims^3 voxels about the surface: which voxels lie
    in the band around it or in front of it, and the band's node lists."""

    def __init__(self, s, dims, lists=True):
        self.dims, self.size = dims, float(np.float32(VOLUME / dims))
        self.params = TsdfParams(dims=(dims,) * 3, voxel_size=self.size, truncation=float(np.float32(5 * self.size)))
        self.grid = voxel_grid(ORIGIN, self.size, (dims,) * 3)
        n = dims ** 3
        a = torch.arange(dims, device=DEV, dtype=F64) + 0.5
        self.sdf = torch.full((n,), -math.inf, device=DEV)
        plane = dims * dims
        for z in range(0, dims, 16):
            Z, Y, X = torch.meshgrid(ORIGIN[2] + a[z:z + 16] * self.size, ORIGIN[1] + a * self.size,
                                     ORIGIN[0] + a * self.size, indexing="ij")
            u, v = s.f * X / Z + s.cx, s.f * Y / Z + s.cy
            ok = (u >= 0) & (u < s.W - 0.5) & (v >= 0) & (v < s.H - 0.5)
            d = s.depth_at(u, v) - Z
            self.sdf[z * plane:(z + 16) * plane] = torch.where(ok, d, torch.full_like(d, -math.inf)).reshape(-1).float()
        if not lists:
            return
        band = (self.sdf.abs() < 6 * self.size).nonzero()[:, 0]
        c = self.centres(band)
        ids, ws = _near(c, s.candidates(s.f * c[:, 0] / c[:, 2] + s.cx, s.f * c[:, 1] / c[:, 2] + s.cy), s.pos,
                        s.radius)
        self.knn = torch.full((n, 4), -1, device=DEV, dtype=torch.int32)
        self.knn_w = torch.zeros(n, 4, device=DEV)
        self.knn[band], self.knn_w[band] = ids.int(), ws.float()

    def centres(self, i):
        d = self.dims
        return torch.stack([(torch.div(i, k, rounding_mode="floor") % d + 0.5) * self.size + o
                            for k, o in zip((1, d, d * d), ORIGIN)], -1).double()

    def voxels(self, g, inside):
        """Records: the truncated distance and a random weight where `inside`."""
        f = torch.zeros(len(self.sdf), 3, device=DEV)
        f[:, 0] = torch.where(inside, (self.sdf / self.params.truncation).clamp(-1, 1), torch.ones_like(self.sdf))
        w = 50 * torch.rand(len(self.sdf), generator=g, device=DEV) + 1e-3
        f[:, 1] = torch.where(inside, w, torch.zeros_like(w))
        f.view(torch.int32)[:, 2] = 0x00808080
        return f


def _pose(g):
    """A small camera motion: camera -> world, and its inverse."""
    a = _randn(g, 3)
    q = _qexp(a / a.norm() * math.radians(0.6))
    T = torch.eye(4, device=DEV, dtype=F64)
    T[:3, :3] = _qrot(q.expand(3, 4), torch.eye(3, device=DEV, dtype=F64)).T
    T[:3, 3] = 0.004 * (_rand(g, 3) - 0.5)
    T = T.cpu()
    return T.numpy().astype(np.float32), torch.linalg.inv(T).numpy().astype(np.float32)


def _observed(g, s):
    """The depth a sensor sees a few millimetres off the model: noise, holes."""
    z = s.z + 0.003 * torch.sin(2 * math.pi * s.u / s.W) + 0.001 * _randn(g, s.H, s.W)
    z = torch.where(_rand(g, s.H, s.W) < 0.01, torch.zeros_like(z), z).float().double()
    n = _normals(s.unproject(z))
    ok = torch.zeros(s.H, s.W, device=DEV, dtype=torch.bool)
    ok[:-1, :-1] = (z[:-1, :-1] > 0) & (z[:-1, 1:] > 0) & (z[1:, :-1] > 0)
    return z, n * ok[..., None]


def _mesh(g, case):
    s = Surface(g, case["width"], case["height"], case["nodes"])
    vol = Volume(s, case["dims"])
    st = case["stride"]
    pts = s.points.view(s.H, s.W, 3)[::st, ::st]
    h, w = pts.shape[:2]
    a = (torch.arange(h - 1, device=DEV)[:, None] * w + torch.arange(w - 1, device=DEV)).reshape(-1)
    m = DeviceMesh.__new__(DeviceMesh)
    m.width, m.height = s.W, s.H
    m.cam = np.array([s.f, s.f, s.cx, s.cy], np.float32)
    m.T_world_cam, m.T_cam_world = _pose(g)
    m.canonical = pts.reshape(-1).float().contiguous()
    m.triangles = torch.cat([torch.stack([a, a + w, a + 1], -1),
                             torch.stack([a + 1, a + w, a + w + 1], -1)]).int().reshape(-1)
    m.num_vertices, m.num_triangles = h * w, 2 * len(a)
    m.grid, m.voxel_knn, m.voxel_knn_w = vol.grid, vol.knn.reshape(-1), vol.knn_w.reshape(-1)
    m.nodes, m.num_nodes = s.nodes(), len(s.pos)
    m.transforms = _warp(g, s.pos, math.radians(3.0), 0.01, 0.5).float().view(torch.uint8).reshape(-1)
    return s, vol, m


def _search_frame(g, s, vol, pose):
    """The search's frame: the model's live maps and the observed depth."""
    f = DeviceCorrFrame.__new__(DeviceCorrFrame)
    f.width, f.height = s.W, s.H
    f.cam = np.array([s.f, s.f, s.cx, s.cy], np.float32)
    f.T_world_cam, f.T_cam_world = pose
    z, n = _observed(g, s)
    f.depth, f.depth_normals = z.float().reshape(-1), n.float().reshape(-1)
    P = s.points.view(s.H, s.W, 3)
    seen = (_rand(g, s.H, s.W) >= 0.02)[..., None]
    f.live_vertices = (P * seen).float().reshape(-1)
    f.live_normals = (_normals(P) * seen).float().reshape(-1)
    o = torch.tensor(ORIGIN, device=DEV, dtype=F64)
    ijk = ((s.points - o) / vol.size).floor().long().clamp(0, vol.dims - 1)
    hit = (ijk[:, 2] * vol.dims + ijk[:, 1]) * vol.dims + ijk[:, 0]
    f.hit_voxel_idx = torch.where(seen.reshape(-1), hit, torch.full_like(hit, -1)).int()
    f.voxel_knn, f.voxel_knn_w, f.num_voxels = vol.knn.reshape(-1), vol.knn_w.reshape(-1), vol.dims ** 3
    hit = f.hit_voxel_idx.long()
    f.pixel_knn = torch.where(hit[:, None] >= 0, vol.knn[hit.clamp_min(0)], -1).int().reshape(-1)
    f.pixel_knn_w = (vol.knn_w[hit.clamp_min(0)] * (hit >= 0)[:, None]).reshape(-1)
    return f


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def _solve_inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "batch":
        return [_sphere_problem(g, n, m, 20.0, 0.03) for n, m in _batch_sizes(case)]
    if case.get("scene") == "sphere":
        return [_sphere_problem(g, case["nodes"], case["corrs"])]
    if case["kind"] == "learned":
        return [_frame_problem(g, case["width"], case["height"], case["nodes"], past=3)]
    return [_frame_problem(g, case["width"], case["height"], case["nodes"], case.get("invalid", 0.0))]


def _solve_params(case):
    # the reference pipeline's production damping and the workloads' ARAP weight
    if case["kind"] == "learned":
        return dict(gn=1, pcg=20, tol=1e-4, consistent=True)
    return dict(gn=case.get("gn", 1), pcg=case["pcg"], tol=0.0 if case.get("scene") == "frame" else 1e-4,
                consistent=False)


def _gradient_inputs(case, seed):
    g = _gen(seed)
    s = Surface(g, 320, 240, case["nodes"])
    n = len(s.nb)
    nbr = torch.full((n, 8), -1, device=DEV, dtype=torch.int64)
    nbr[:, :s.nb.shape[1]] = s.nb
    nbr = torch.cat([torch.where(nbr >= 0, nbr + k * n, nbr) for k in range(case["frames"])]).int()
    x = torch.randn(len(nbr), learned.IN, generator=g, device=DEV)
    y = torch.randn(len(nbr), learned.OUT, generator=g, device=DEV)
    w = learned.init_weights(int(seed) % 1000).copy()
    w[-390:] += np.random.default_rng(int(seed)).normal(scale=0.1, size=390).astype(np.float32)
    return nbr, x, y, w


_STREAMS = []


def _stream():
    """The stream that the program runs its solves on: off the legacy stream
    they replay their launch sequence, one after another as its frames come."""
    if not _STREAMS:
        _STREAMS.append(torch.cuda.Stream())
    return _STREAMS[0]


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind in ("solve", "batch", "linearize", "learned"):
        ps = _solve_inputs(case, seed)
        q = _solve_params(case)
        st["problems"] = ps
        st["solver"] = GaussNewtonSolver(
            Params(gn_iterations=q["gn"], pcg_iterations=q["pcg"], pcg_tolerance=q["tol"], lambda_smooth=10.0,
                   lambda_damping=1.0),
            max_nodes=sum(p.num_nodes for p in ps), max_corrs=sum(p.num_corrs for p in ps))
        st["solver"].set_arap_consistent(q["consistent"])
        st["T"] = [p.init_transforms.clone() for p in ps]
        st["dx"] = torch.zeros(6 * ps[0].num_nodes, device=DEV)
        if kind == "learned":
            st["net"] = learned.MPNN(ps[0].num_nodes, np.load(learned.WEIGHTS))
    elif kind == "gradients":
        nbr, st["x"], st["y"], w = _gradient_inputs(case, seed)
        st["net"] = learned.MPNN(len(nbr), w)
        st["net"].set_graph(nbr)
    elif kind in ("predict", "linesearch"):
        g = _gen(seed)
        s, vol, m = _mesh(g, case)
        st.update(mesh=m, raster=LiveSurfaceRaster(s.W, s.H), warped=torch.empty_like(m.canonical))
        if kind == "linesearch":
            n = m.num_nodes
            dx = torch.cat([_smooth(g, s.pos, 0.01, 0.5), _smooth(g, s.pos, 0.003, 0.5)], 1)
            st.update(frame=_search_frame(g, s, vol, (m.T_world_cam, m.T_cam_world)), T=m.transforms.clone(),
                      search=CorrespondenceSearch(s.W, s.H), ls=LineSearch(n), dx=dx.float().reshape(-1),
                      prm=LineSearchParams(max_update_rot=CLAMPS[0], max_update_trans=CLAMPS[1]),
                      cprm=CorrParams(search_radius_px=case["radius"]), base=(0.004, s.W * s.H // 2))
    elif kind == "search":
        g = _gen(seed)
        s = Surface(g, case["width"], case["height"], max(64, min(2048, case["width"] * case["height"] // 150)))
        st.update(frame=_search_frame(g, s, Volume(s, 128), _pose(g)), search=CorrespondenceSearch(s.W, s.H),
                  prm=CorrParams(dist_threshold=case["dist"], angle_threshold=case["angle"],
                                 search_radius_px=case["radius"]))
    else:
        st.update(_volume_inputs(case, seed))
        st["vol"] = TSDFVolume(st["params"])
        st["vol"].voxels.copy_(st["voxels"].view(torch.uint8).reshape(-1))
        if kind == "integrate":
            st["vol"].integrate(torch.zeros_like(st["depth"]), st["cam"], st["pose"], **st["warp"])
        del st["voxels"]
    st["stream"] = _stream()
    torch.cuda.synchronize()
    return st


def _volume_inputs(case, seed):
    g = _gen(seed)
    s = Surface(g, case["width"], case["height"], case["nodes"])
    vol = Volume(s, case["dims"], lists=case["kind"] == "integrate")
    out = dict(params=vol.params, nodes=s.nodes(), num_nodes=len(s.pos), volume=vol, pos=s.pos, radius=s.radius)
    if case["kind"] == "voxelknn":
        # what an integrated frame leaves: data in front of the surface and in the band behind it
        out["voxels"] = vol.voxels(g, vol.sdf >= -vol.params.truncation)
        out["knn"] = torch.empty(4 * vol.dims ** 3, dtype=torch.int32, device=DEV)
        out["knn_w"] = torch.empty(4 * vol.dims ** 3, device=DEV)
        del out["volume"].sdf
        return out
    near = vol.sdf.abs() < 15 * vol.size
    out["voxels"] = vol.voxels(g, near)
    z, _ = _observed(g, s)
    bad = _rand(g, s.H, s.W)
    z = torch.where(bad < 0.001, torch.full_like(z, -0.5), z)
    out.update(depth=z.float().reshape(-1), cam=s.cam, pose=_pose(g)[0], surface=s)
    T = _warp(g, s.pos, math.radians(3.0), 0.01, 0.5).float()
    counts = torch.randint(0, 7, (vol.dims ** 3,), generator=g, device=DEV, dtype=torch.int32) * near
    out["warp"] = {}
    if case["warp"]:
        out["warp"] = dict(nodes=out["nodes"], transforms=T.view(torch.uint8).reshape(-1), num_nodes=len(s.pos),
                           voxel_knn=vol.knn.reshape(-1), voxel_knn_w=vol.knn_w.reshape(-1),
                           voxel_opt_counts=counts.int(), min_opt_count=3)
    return out


def _f32(b):
    return b.view(torch.float32)


def run(st):
    kind = st["kind"]
    if kind in ("solve", "batch", "learned"):
        ps, T, side = st["problems"], st["T"], st["stream"]
        with torch.cuda.stream(side):
            for t, p in zip(T, ps):
                t.copy_(p.init_transforms)
            if kind == "solve":
                st["solver"].gn_solve(ps[0], T[0], *CLAMPS, stats=False, stream=side)
            elif kind == "batch":
                st["solver"].gn_solve_batched(ps, T, *CLAMPS, stats=False, stream=side)
            else:
                learned.solve_learned(st["solver"], st["net"], ps[0], T[0], ps[0].history, *CLAMPS, stats=False)
        return [_f32(t) for t in T]
    if kind == "linearize":
        p = st["problems"][0]
        return st["solver"].solve(p.corrs, p.num_corrs, p.nodes, p.init_transforms, p.num_nodes, st["dx"])
    if kind == "gradients":
        loss, grad = st["net"].gradients(st["x"], st["y"])
        return dict(loss=float(loss), grad=grad)
    if kind == "search":
        s, f = st["search"], st["frame"]
        n = s.find_correspondences(f, st["prm"], use_voxels=st["case"]["voxels"])
        return dict(valid=n, records=s.corrs)
    if kind == "predict":
        r = st["raster"]
        r.predict(st["mesh"], st["warped"])
        return dict(warped=st["warped"], vertices=r.live_vertices, normals=r.live_normals, voxel=r.hit_voxel_idx)
    if kind == "linesearch":
        side, T, f, r = st["stream"], st["T"], st["frame"], st["raster"]
        with torch.cuda.stream(side):
            T.copy_(st["mesh"].transforms)
            res = st["ls"].run(r, st["search"], st["mesh"], f, T, st["dx"], *st["base"], st["prm"], st["cprm"],
                               st["warped"], stream=side)
        return dict(scale=res["best_scale"], valid=np.array(res["trial_valid"]), rmse=np.array(res["trial_rmse"]),
                    T=_f32(T), vertices=f.live_vertices, voxel=f.hit_voxel_idx, records=st["search"].corrs)
    if kind == "integrate":
        st["vol"].integrate(st["depth"], st["cam"], st["pose"], **st["warp"])
        v = st["vol"].fields()
        return dict(tsdf=v[:, 0], weight=v[:, 1])
    ids, ws = st["vol"].compute_voxel_knn(st["nodes"], st["num_nodes"], st["knn"], st["knn_w"])
    return dict(ids=ids, weights=ws)


def work(case):
    kind = case["kind"]
    px = case.get("width", 0) * case.get("height", 0)
    if kind in ("solve", "batch", "linearize", "learned"):
        if kind == "batch":
            sizes = _batch_sizes(case)
        else:
            sizes = [(case["nodes"], case.get("corrs", px))]
        n, m = sum(a for a, _ in sizes), sum(b for _, b in sizes)
        gn, pcg = (1, 20) if kind == "learned" else (case.get("gn", 1), case["pcg"])
        skin = 0 if kind == "linearize" else 12
        return {"bytes": (76 + skin) * m + (96 + 64) * n,
                "flops": gn * ((250 + 2 * 10 * 21) * m + pcg * n * 10 * 72 + 2000 * n)}
    if kind == "gradients":
        n = case["nodes"] * case["frames"]
        return {"bytes": n * (learned.IN + learned.OUT + 8) * 4 + 8 * learned.PARAMS, "flops": 6 * n * learned.PARAMS}
    if kind == "search":
        r = case["radius"]
        return {"bytes": px * (24 + 16 + 76 + 36), "flops": 10 * px * (2 * r + 1) ** 2}
    if kind == "predict":
        v = px // case["stride"] ** 2
        return {"bytes": v * (24 + 32) + 2 * v * 12 + px * 28 + 128 * case["nodes"], "flops": 200 * v + 100 * px}
    if kind == "linesearch":
        v, r = px // case["stride"] ** 2, case["radius"]
        return {"bytes": v * (24 + 32) + 2 * v * 12 + px * (16 + 28 + 76 + 36),
                "flops": 10 * (200 * v + 100 * px + 10 * px * (2 * r + 1) ** 2)}
    n = case["dims"] ** 3
    if kind == "integrate":
        # the counts of every voxel, the lists and both fields of those in the band
        band = int(0.04 * n)
        return {"bytes": (4 * n if case["warp"] else 0) + band * (32 + 16) + 4 * px, "flops": 200 * band + 4 * n}
    return {"bytes": 44 * n + 16 * case["nodes"], "flops": 8 * 0.12 * n * 64}


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------


def _c(v):
    return float(np.float32(v))


def _huber(r, delta):
    a = r.abs()
    return torch.where(a <= delta, torch.ones_like(a), delta / a.clamp_min(1e-300))


def _rot_plain(T, p):
    return _qrot(T[:, :4], p) + 2 * _qmul(T[:, 4:], _qconj(T[:, :4]))[:, :3]


def _exp_se3(tw):
    """[N, 6] twists -> (rotation quaternion, translation)."""
    w, v = tw[:, :3], tw[:, 3:]
    th = w.norm(dim=-1, keepdim=True).clamp_min(1e-12)
    a = (1 - torch.cos(th)) / th ** 2
    b = (th - torch.sin(th)) / th ** 3
    small = th < 1e-4
    a = torch.where(small, 0.5 - th ** 2 / 24, a)
    b = torch.where(small, 1 / 6 - th ** 2 / 120, b)
    c = torch.linalg.cross(w, v)
    return _qexp(w), v + a * c + b * torch.linalg.cross(w, c)


class _System:
    """The Gauss-Newton system of a problem, assembled and solved in 64 bits."""

    def __init__(self, p, q):
        self.q = q
        f = _f32(p.corrs).view(-1, 19)
        i = p.corrs.view(torch.int32).view(-1, 19)
        self.src, self.dst, self.nrm = f[:, 0:3].double(), f[:, 3:6].double(), f[:, 6:9].double()
        self.ids, self.ws = i[:, 9:13].long(), f[:, 13:17].double()
        self.weight, self.valid = f[:, 17].double(), (i[:, 18] & 255) != 0
        self.canon = p.canon.double()
        nf, ni = _f32(p.nodes).view(-1, 24), p.nodes.view(torch.int32).view(-1, 24)
        self.pos, n = nf[:, :3].double(), len(nf)
        self.n = n
        nb, nw, cnt = ni[:, 7:15].long(), nf[:, 15:23].double(), ni[:, 23]
        ok = (torch.arange(8, device=DEV)[None] < cnt[:, None]) & (nb >= 0) & (nb < n)
        row = torch.arange(n, device=DEV)[:, None].expand(n, 8)
        d = torch.arange(n, device=DEV)
        keys = torch.cat([d * n + d, (row * n + nb)[ok], (nb * n + row)[ok]]).unique()
        self.rows, self.cols = torch.div(keys, n, rounding_mode="floor"), keys % n
        self.block = torch.full((n * n,), -1, device=DEV, dtype=torch.int32)
        self.block[keys] = torch.arange(len(keys), device=DEV, dtype=torch.int32)
        e = ok & (nb > row)
        self.ei, self.ej, self.ew = row[e], nb[e], nw[e].clamp_min(_c(0.05))

    def at(self, i, j):
        return self.block[i * self.n + j].long()

    def edges(self, T):
        """As rigid as possible, each edge once, from its lower node: the
        residuals, their weights and the two ends' images of the upper node."""
        i, j = self.ei, self.ej
        xi, xj = self.pos[i], self.pos[j]

        def centred(T, p, c):
            return _rot_plain(T, p) + c - _qrot(T[:, :4], c)

        a, c, d = centred(T[i], xj, xi), centred(T[i], xi, xi), centred(T[j], xj, xj)
        rest = (xi - xj).norm(dim=-1)
        strain = ((c - d).norm(dim=-1) - rest).abs() / rest.clamp_min(_c(1e-6))
        r = a - d
        el = 10.0 * self.ew * _huber(r.norm(dim=-1), _c(0.05)) * torch.exp(-(strain / 0.25) ** 2)
        return r, torch.where(el <= _c(1e-8), torch.zeros_like(el), el), a, d

    def assemble(self, T, src):
        A = torch.zeros(len(self.rows), 36, device=DEV, dtype=F64)
        b = torch.zeros(self.n, 6, device=DEV, dtype=F64)
        res = (self.nrm * (src - self.dst)).sum(-1)
        fw = self.weight.clamp_min(0) * _huber(res, _c(0.2))
        on = self.valid & (fw > _c(1e-8))
        for s in torch.arange(len(src), device=DEV)[on].split(1 << 18):
            J, ok = [], []
            for k in range(4):
                i, w = self.ids[s, k], self.ws[s, k]
                ok.append((i >= 0) & (i < self.n) & (w > _c(1e-8)))
                i = i.clamp(0, self.n - 1)
                J.append(w[:, None] * torch.cat([torch.linalg.cross(src[s] - self.pos[i], self.nrm[s]),
                                                 self.nrm[s]], -1))
                b.index_add_(0, i[ok[k]], -(fw[s] * res[s])[ok[k], None] * J[k][ok[k]])
            for x in range(4):
                for y in range(4):
                    m = ok[x] & ok[y]
                    q = self.at(self.ids[s, x].clamp(0, self.n - 1), self.ids[s, y].clamp(0, self.n - 1))
                    m &= q >= 0
                    A.index_add_(0, q[m], (fw[s][m, None, None] * J[x][m][:, :, None] * J[y][m][:, None, :]
                                           ).reshape(-1, 36))
        r, el, a, d = self.edges(T)
        i, j, xi, xj = self.ei, self.ej, self.pos[self.ei], self.pos[self.ej]

        def jac(p):
            z = torch.zeros_like(p[:, 0])
            J = torch.stack([torch.stack([z, p[:, 2], -p[:, 1]], -1), torch.stack([-p[:, 2], z, p[:, 0]], -1),
                             torch.stack([p[:, 1], -p[:, 0], z], -1)], 1)
            J = -J if self.q["consistent"] else J
            return torch.cat([J, torch.eye(3, device=DEV, dtype=F64).expand(len(p), 3, 3)], 1)

        Ji, Jj = jac(a - xi), jac(d - xj)
        for x, y, Jx, Jy, sign in ((i, i, Ji, Ji, 1), (j, j, Jj, Jj, 1), (i, j, Ji, Jj, -1), (j, i, Jj, Ji, -1)):
            A.index_add_(0, self.at(x, y), (sign * el[:, None, None] * (Jx @ Jy.transpose(1, 2))).reshape(-1, 36))
        b.index_add_(0, i, -el[:, None] * (Ji @ r[..., None])[..., 0])
        b.index_add_(0, j, el[:, None] * (Jj @ r[..., None])[..., 0])
        # relative damping with its floors
        k = torch.arange(self.n, device=DEV)
        D = A[self.at(k, k)].view(-1, 6, 6)
        dg = torch.diagonal(D, dim1=1, dim2=2)
        floor = torch.tensor([1e-3] * 3 + [1e-2] * 3, device=DEV, dtype=F64)
        dg += torch.maximum(dg.abs(), floor)  # lambda_damping = 1
        A[self.at(k, k)] = D.reshape(-1, 36)
        return A.view(-1, 6, 6), b, D

    def pcg(self, A, b, D):
        eye = torch.eye(6, device=DEV, dtype=F64)
        M = D + _c(1e-4) * eye
        L, bad = torch.linalg.cholesky_ex(M)
        inv = torch.cholesky_inverse(L)
        flat = torch.diag_embed(1 / (torch.diagonal(M, dim1=1, dim2=2) + _c(1e-6)))
        inv = torch.where((bad > 0)[:, None, None], flat, inv)

        def pre(r):
            return (inv @ r[..., None])[..., 0]

        def mul(p):
            y = torch.zeros_like(p)
            return y.index_add_(0, self.rows, (A @ p[self.cols][..., None])[..., 0])

        x, r = torch.zeros_like(b), b.clone()
        z = pre(r)
        p, rz = z.clone(), float((r * z).sum())
        for _ in range(self.q["pcg"]):
            Ap = mul(p)
            pAp = float((p * Ap).sum())
            if abs(pAp) < _c(1e-12):
                break
            x, r = x + rz / pAp * p, r - rz / pAp * Ap
            if float(r.norm()) < self.q["tol"]:
                break
            z = pre(r)
            new = float((r * z).sum())
            p, rz = z + new / rz * p, new
        return x

    def solve(self, T):
        for _ in range(self.q["gn"]):
            src = _skin(self.canon, self.ids, self.ws, self.pos, T)[0]
            dx = self.pcg(*self.assemble(T, src))
            T = _twist(T, dx, *CLAMPS)
        return T

    def residuals(self, T):
        src = _skin(self.canon, self.ids, self.ws, self.pos, T)[0]
        return (self.nrm * (src - self.dst)).sum(-1)

    def energy(self, T):
        res = self.residuals(T)
        fw = self.weight.clamp_min(0) * _huber(res, _c(0.2)) * self.valid
        r, el = self.edges(T)[:2]
        return float((fw * res ** 2).sum() + (el * (r ** 2).sum(-1)).sum())


def _twist(T, dx, rot, trans):
    w, v = dx[:, :3], dx[:, 3:]
    w = w * (rot / w.norm(dim=-1, keepdim=True).clamp_min(rot))
    v = v * (trans / v.norm(dim=-1, keepdim=True).clamp_min(trans))
    q, t = _exp_se3(torch.cat([w, v], -1))
    D = _dq(q, t)
    real = _qmul(D[:, :4], T[:, :4])
    dual = _qmul(D[:, :4], T[:, 4:]) + _qmul(D[:, 4:], T[:, :4])
    n = real.norm(dim=-1, keepdim=True)
    return torch.cat([real / n, dual / n], -1)


def _network64(theta, x, nbr):
    """The network in 64 bits on the 16-bit parameters and inputs it holds."""
    P, o = [], 0
    for _, shape in learned.SHAPES:
        k = int(np.prod(shape))
        P.append(theta[o:o + k].view(shape))
        o += k
    ok = (nbr >= 0).double()
    deg = ok.sum(1, keepdim=True).clamp_min(1)
    h = x.bfloat16().double()
    for k in range(3):
        m = (h[nbr.clamp_min(0).long()] * ok[..., None]).sum(1) / deg
        h = torch.relu(torch.cat([h, m], 1) @ P[2 * k].T + P[2 * k + 1])
    return h @ P[6].T + P[7] + x[:, :6].double()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "linearize"):
        p = _solve_inputs(case, seed)[0]
        s = _System(p, _solve_params(case))
        T = _f32(p.init_transforms).view(-1, 8).double()
        if kind == "linearize":
            return s.pcg(*s.assemble(T, s.src)).reshape(-1)
        return [s.solve(T).reshape(-1)]
    if kind == "batch":
        if sum(m for _, m in _batch_sizes(case)) > 4_000_000:
            return None  # minutes in 64 bits
        out = []
        for p in _solve_inputs(case, seed):
            s = _System(p, _solve_params(case))
            out.append(s.solve(_f32(p.init_transforms).view(-1, 8).double()).reshape(-1))
        return out
    if kind == "gradients":
        nbr, x, y, w = _gradient_inputs(case, seed)
        theta = torch.from_numpy(w).to(DEV).bfloat16().double().requires_grad_(True)
        loss = ((_network64(theta, x, nbr) - y.double()) ** 2).mean()
        loss.backward()
        return dict(loss=float(loss.detach()), grad=theta.grad)
    if kind == "predict":
        g = _gen(seed)
        s, vol, m = _mesh(g, case)
        v = m.canonical.view(-1, 3)
        # the voxels as 32-bit arithmetic finds them
        o = torch.tensor(ORIGIN, device=DEV, dtype=torch.float32)
        ijk = ((v - o) / torch.tensor(vol.size, device=DEV, dtype=torch.float32)).floor().long()
        i = (ijk[:, 2] * vol.dims + ijk[:, 1]) * vol.dims + ijk[:, 0]
        out = _skin(v.double(), vol.knn[i].long(), vol.knn_w[i].double(), s.pos,
                    _f32(m.transforms).view(-1, 8).double())[0]
        # the maps follow from which triangle 32-bit rounding puts in front
        return dict(warped=out.reshape(-1), vertices=None, normals=None, voxel=None)
    if kind == "learned":
        return [_exact_learned(case, seed).reshape(-1)]
    if kind == "voxelknn":
        return dict(ids=None, weights=_exact_lists(case, seed))
    # a search, a line search and an integration choose a candidate, a pixel or
    # a triangle by differences that 32 bits round: their results are the choice's
    return None


def _exact_lists(case, seed):
    st = _volume_inputs(case, seed)
    vol, pos, n = st["volume"], st["pos"], case["dims"] ** 3
    out = torch.zeros(n, 4, device=DEV, dtype=F64)
    on = (st["voxels"][:, 1] > 0).nonzero()[:, 0]
    r = torch.full((len(pos),), max(st["radius"], 1e-6), device=DEV, dtype=F64)
    for i in on.split(1 << 16):
        c = vol.centres(i)
        d, o = torch.cdist(c.float(), pos.float(), compute_mode="donot_use_mm_for_euclid_dist").topk(
            min(8, len(pos)), largest=False)
        d = ((pos[o] - c[:, None]) ** 2).sum(-1)
        d, k = d.topk(4, largest=False)
        out[i] = _weights(d, r[0])
    return out.reshape(-1)


def _exact_learned(case, seed):
    p = _solve_inputs(case, seed)[0]
    s = _System(p, _solve_params(case))
    hist = _f32(p.history).view(3, -1, 8).double()
    T = _f32(p.init_transforms).view(-1, 8).double()
    chain = [T] + list(hist)
    cols = []
    for a, b in zip(chain[:-1], chain[1:]):
        # the increment D with a = D b, as node-centred dual quaternions
        q = _qmul(a[:, :4], _qconj(b[:, :4]))
        q = torch.where(q[:, 3:] < 0, -q, q)
        n = q[:, :3].norm(dim=-1, keepdim=True)
        w = q[:, :3] * (2 * torch.atan2(n, q[:, 3:]) / n.clamp_min(1e-30))
        ta, tb = (2 * _qmul(x[:, 4:], _qconj(x[:, :4]))[:, :3] for x in (a, b))
        cols += [w * _lib.CF_MPNN_ROT_SCALE, (ta - _qrot(q, tb)) * _lib.CF_MPNN_TRANS_SCALE]
    res = s.residuals(T).abs() * 1000.0
    tot, top, cnt = (torch.zeros(s.n, device=DEV, dtype=F64) for _ in range(3))
    for k in range(4):
        m = s.valid & (s.ws[:, k] > _c(1e-8))
        i = s.ids[m, k]
        tot.index_add_(0, i, res[m])
        cnt.index_add_(0, i, torch.ones_like(res[m]))
        top.scatter_reduce_(0, i, res[m], "amax")
    x = torch.cat(cols + [(tot / cnt.clamp_min(1))[:, None], top[:, None]], 1)
    ni = p.nodes.view(torch.int32).view(-1, 24)
    theta = torch.from_numpy(np.load(learned.WEIGHTS)).to(DEV).bfloat16().double()
    d = _network64(theta, x, ni[:, 7:15])
    w, v = d[:, :3] / _lib.CF_MPNN_ROT_SCALE, d[:, 3:] / _lib.CF_MPNN_TRANS_SCALE
    q, t = _qexp(w), 2 * _qmul(T[:, 4:], _qconj(T[:, :4]))[:, :3]
    start = _dq(_qmul(q, T[:, :4]), _qrot(q, t) + v)
    return s.solve(start if s.energy(start) <= s.energy(T) else T)
