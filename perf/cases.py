"""Performance cases of the framework: what a user's program has it do, through its public entry points.

Kinds of case:

* ``reconstruct``  a whole ``jspsr.reconstruct`` call on an oriented point cloud.  The solutions of all
  levels and the field at the mesh's samples are returned; the triangles are not, because a sample whose
  field value rounds to the other side of zero changes their number (``mesh`` returns triangles).
* ``field``        the solved field and its gradient at query points (rendering, losses, normals).
* ``mesh``         multi-level dual marching cubes over given leaf cells for a given field.
* ``solve``        an assembled level system solved to FP64 accuracy (the direct solve of the class API).
* ``learned``      a training step of the learned-basis form: trees, geometry, forward, adjoint.
* ``conv``         a sparse convolution layer of the network, forward or forward and backward.
* ``sdf``          ground-truth signed distances (and neighbours) from an oriented point cloud.

The points of a case are the same for every seed wherever the sizes of its outputs follow from them; the seed
then sets their order, the normals, the features, the weights and the right-hand sides.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "neural-galerkin_b200"))

DEV = "cuda"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest request of a serving stream: launches and synchronisations dominate
        dict(name="reconstruct_2k", kind="reconstruct", cloud="mixed", n=2003, voxel=1 / 64, depth=4, share=0.5),
        # an ordinary request of a serving stream
        dict(name="reconstruct_50k", kind="reconstruct", cloud="mixed", n=50000, voxel=1 / 256, depth=4, share=0.5),
        # the benchmark's reconstruction
        dict(name="reconstruct_300k", kind="reconstruct", cloud="superquadrics", n=300000, voxel=1 / 512, depth=4,
             share=0.85),
        # the largest scene: a scanned room at 1 cm, eleven levels
        dict(name="reconstruct_room_5m", kind="reconstruct", cloud="room", n=5000000, voxel=0.01, depth=11, share=0.98),
        # field and normals at a million points of a solved reconstruction
        dict(name="field_1m", kind="field", n=100000, voxel=1 / 256, depth=4, share=0.85, queries=1000003),
        # the mesh of a benchmark-sized hierarchy
        dict(name="mesh_300k", kind="mesh", n=300000, voxel=1 / 512, depth=4, share=0.85),
        # the direct solve of one level's system, some 160,000 rows
        dict(name="solve_160k", kind="solve", n=30011, voxel=1 / 256),
        # a training step on a small batch of shapes
        dict(name="learned_4", kind="learned", shapes=4, n=3000, queries=20000, voxel=1 / 128, depth=3),
        # inference through the network's middle layer on the benchmark's finest level
        dict(name="conv_bf16_1m", kind="conv", n=300000, voxel=1 / 512, kernel=3, cin=64, cout=64, dtype="bf16",
             train=False),
        # a training step of that layer in half precision
        dict(name="conv_f16_train_250k", kind="conv", n=100003, voxel=1 / 256, kernel=3, cin=64, cout=64, dtype="f16",
             train=True),
        # the first layer of a network that is trained in single precision
        dict(name="conv_f32_train_30k", kind="conv", n=10000, voxel=1 / 128, kernel=3, cin=16, cout=32, dtype="f32",
             train=True),
        # the training loop's ground truth
        dict(name="sdf_100k", kind="sdf", n=60000, queries=100000, k=8, want="sdf"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reconstruct", "reconstruct", "field", "mesh", "solve", "learned", "conv", "conv", "sdf"])
    if kind == "reconstruct":
        return dict(kind=kind, cloud=rng.choice(["mixed", "mixed", "superquadrics", "torus"]), n=_log(rng, 1000, 500000),
                    voxel=2.0 ** -rng.randint(6, 9), depth=rng.choice([3, 4, 4, 5]), share=rng.choice([0.5, 0.85]))
    if kind == "field":
        return dict(kind=kind, n=_log(rng, 3000, 300000), voxel=2.0 ** -rng.randint(6, 9), depth=rng.choice([3, 4, 5]),
                    share=rng.choice([0.5, 0.85]), queries=_log(rng, 1000, 2000000))
    if kind == "mesh":
        return dict(kind=kind, n=_log(rng, 1000, 500000), voxel=2.0 ** -rng.randint(6, 9), depth=rng.choice([3, 4, 5]),
                    share=rng.choice([0.5, 0.85]))
    if kind == "solve":
        return dict(kind=kind, n=_log(rng, 500, 100000), voxel=2.0 ** -rng.randint(6, 9))
    if kind == "learned":
        return dict(kind=kind, shapes=rng.randint(1, 6), n=_log(rng, 1000, 6000), queries=_log(rng, 2000, 40000),
                    voxel=1 / 128, depth=3)
    if kind == "conv":
        dtype = rng.choice(["f16", "bf16", "f32"])
        wide = [16, 32, 48, 64] if dtype == "f32" else [16, 32, 64, 96, 128, 256]
        return dict(kind=kind, n=_log(rng, 2000, 30000 if dtype == "f32" else 300000), voxel=2.0 ** -rng.randint(7, 9),
                    kernel=rng.choice([3, 3, 2]), cin=rng.choice([4] + wide), cout=rng.choice(wide), dtype=dtype,
                    train=rng.random() < 0.5)
    return dict(kind=kind, n=_log(rng, 2000, 60000), queries=_log(rng, 1000, 100000), k=rng.choice([1, 4, 8, 16]),
                want=rng.choice(["sdf", "knn"]))


# ----------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _torus(n, seed, noise=0.002, R=0.31, r=0.13):
    """Oriented points on a torus, with position noise."""
    g = _gen(seed)
    u = _rand(g, n) * 2 * math.pi
    v = _rand(g, n) * 2 * math.pi
    nrm = torch.stack([v.cos() * u.cos(), v.cos() * u.sin(), v.sin()], 1)
    ring = torch.stack([u.cos(), u.sin(), torch.zeros_like(u)], 1)
    xyz = R * ring + r * nrm + noise * _randn(g, n, 3)
    return xyz.float().contiguous(), nrm.float().contiguous()


def _cloud(case):
    from jspsr import synthetic
    n = case["n"]
    if case["cloud"] == "torus":
        return _torus(n, n)
    if case["cloud"] == "mixed":
        return synthetic.serving_request_device(dict(n=n, seed=n), DEV)
    if case["cloud"] == "room":
        xyz, nrm = synthetic.room(n=n, seed=0)
    else:
        xyz, nrm, _ = synthetic.superquadrics(n, k=4, seed=0)
    return torch.from_numpy(xyz).to(DEV), torch.from_numpy(nrm).to(DEV)


def _noisy(nrm, g):
    """Unit normals with the noise of an estimate."""
    nrm = nrm.double() + 0.02 * _randn(g, *nrm.shape)
    return (nrm / nrm.norm(dim=1, keepdim=True)).float().contiguous()


def _cloud_inputs(case, seed):
    """The case's points in an order, and with normal noise, of the seed's."""
    xyz, nrm = _cloud(case)
    g, at = _gen(seed), np.random.default_rng(int(seed)).integers(len(xyz))
    return xyz.roll(int(at), 0).contiguous(), _noisy(nrm.roll(int(at), 0), g)


def _bspline(x):
    a = x.abs()
    return torch.where(a < 0.5, 1.5 - 2 * x * x, torch.where(a < 1.5, (a - 1.5) ** 2, torch.zeros_like(x)))


def _dbspline(x):
    a = x.abs()
    return torch.where(a < 0.5, -4 * x, torch.where(a < 1.5, 2 * (a - 1.5) * torch.sign(x), torch.zeros_like(x)))


def _bits(device=DEV):
    b = torch.arange(8, device=device)
    return torch.stack([b >> 2 & 1, b >> 1 & 1, b & 1], 1)


def _density(xyz, voxel):
    """The kernel density that assigns points to levels, in 64 bits."""
    q = xyz.double() / (4 * voxel)
    d = q.floor()
    rel = q - d - 0.5
    loc, sg = rel.abs(), torch.sign(rel)
    lo = d.min(0).values - 2
    dims = (d.max(0).values + 3 - lo).long().tolist()
    grid = torch.zeros(dims[0] * dims[1] * dims[2], dtype=torch.float64, device=DEV)

    def flat(c):
        c = (c - lo).long()
        return (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    for b in _bits().double():
        w = torch.where(b > 0, loc, 1 - loc).prod(1)
        grid.index_add_(0, flat(d + b * sg), w)
    out = torch.zeros(xyz.shape[0], dtype=torch.float64, device=DEV)
    for k in range(27):
        o = torch.tensor([k // 9 - 1, k // 3 % 3 - 1, k % 3 - 1], dtype=torch.float64, device=DEV)
        out += _bspline(q - (d + o + 0.5)).prod(1) * grid[flat(d + o)]
    return out / 16


def _min_density(xyz, voxel, depth, share):
    """The layering threshold that puts ``share`` of the points on the finest level, taken in the middle of
    a gap between densities, so that the last bits of a density move no point to another level."""
    rho = torch.sort(torch.log2(_density(xyz, voxel)) / 2).values
    n = rho.numel()
    at = int(n * (1 - share))
    half = max(8, min(4096, n // 50))
    lo, hi = max(at - half, 0), min(at + half, n - 2)
    t = 0.5 * (rho[lo:hi] + rho[lo + 1:hi + 1])
    clear = torch.full_like(t, math.inf)
    for k in range(max(depth - 1, 1)):
        i = torch.searchsorted(rho, t - k)
        clear = torch.minimum(clear, (rho[i.clamp(max=n - 1)] - (t - k)).abs())
        clear = torch.minimum(clear, (rho[(i - 1).clamp(min=0)] - (t - k)).abs())
    return float(4.0 ** t[clear.argmax()])


def _corners(xyz, voxel, stride):
    """The eight trilinear corner cells of every point, in the library's FP32 quantisation."""
    q = xyz * float(np.float32(1.0) / np.float32(voxel))
    d = (q / stride).floor() * stride
    sg = torch.sign((q - d) - 0.5 * stride)
    return (d[:, None] + _bits()[None] * sg[:, None] * stride).reshape(-1, 3).long()


def _pack(c):
    c = c + (1 << 19)
    return (c[..., 0] << 42) | (c[..., 1] << 21) | c[..., 2]


def _unpack(k):
    m = (1 << 21) - 1
    return torch.stack([k >> 42, (k >> 21) & m, k & m], -1) - (1 << 19)


def _levels(xyz, voxel, depth, min_density):
    """Sorted keys of every level's voxels."""
    lv = (-torch.floor(torch.log2(_density(xyz, voxel) / min_density) / 2)).clamp(0, depth - 1)
    return [torch.unique(_pack(_corners(xyz[lv <= d], voxel, 2 ** d))) for d in range(depth)]


def _coefficients(coords, stride, voxel, seed):
    """Coefficients like those of a solved level: a smooth function of the voxel's position, with detail."""
    p = (coords.double() + 0.5 * stride) * voxel
    g = np.random.default_rng(int(seed) + stride)
    a = torch.tensor(g.normal(0, 1, (3, 3)) * [[9.0], [27.0], [0.3 / voxel / stride]], device=DEV)
    w = torch.tensor([0.05, 0.02, 0.005], dtype=torch.float64, device=DEV)
    return ((torch.sin(p @ a.T) * w).sum(1) / stride).float()


def _leaf_cells(xyz, voxel, depth, min_density):
    """Conformal leaf cells per level, int32: the children of a level's parent cells that no finer level covers."""
    keys = _levels(xyz, voxel, depth, min_density)
    out, finer = [], None
    for d in range(depth):
        c, s = _unpack(keys[d]), 2 ** d
        parents = torch.unique(_pack(torch.div(c, 2 * s, rounding_mode="floor") * (2 * s)))
        if d < depth - 1:
            c = (_unpack(parents)[:, None] + _bits()[None] * s).reshape(-1, 3)
        if finer is not None:
            c = c[~torch.isin(_pack(c), finer)]
        out.append(c.int().contiguous())
        finer = parents
    return out


def _kernel_map(case):
    """Coordinates and the (input, output) pairs of every offset of a 3^3 layer, or of a 2^3 stride-2 layer."""
    xyz, _ = _torus(case["n"], case["n"])
    src = torch.unique(_pack(_corners(xyz, case["voxel"], 1)))
    if case["kernel"] == 3:
        tgt, offs = src, [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]
    else:
        tgt = torch.unique(_pack(torch.div(_unpack(src), 2, rounding_mode="floor") * 2))
        offs = [(x, y, z) for x in (0, 1) for y in (0, 1) for z in (0, 1)]
    pairs, sizes = [], []
    for x, y, z in offs:
        want = tgt + ((x << 42) + (y << 21) + z)
        at = torch.searchsorted(src, want).clamp(max=src.numel() - 1)
        hit = torch.nonzero(src[at] == want)[:, 0]
        pairs.append(torch.stack([at[hit], hit], 1).int())
        sizes.append(hit.numel())
    return src.numel(), tgt.numel(), torch.cat(pairs).contiguous(), torch.tensor(sizes, dtype=torch.int32)


def _conv_inputs(case, seed):
    n_in, n_out, maps, sizes = _kernel_map(case)
    g, dt = _gen(seed + 1), DTYPES[case["dtype"]]
    K = case["kernel"] ** 3
    x = _randn(g, n_in, case["cin"]).to(dt)
    w = (_randn(g, K, case["cin"], case["cout"]) / math.sqrt(0.6 * K * case["cin"])).to(dt)
    gy = _randn(g, n_out, case["cout"]).to(dt)
    return n_in, n_out, maps, sizes, x, w, gy


def _system(case, seed):
    """A level's screened stiffness matrix (CSR, FP32 values) over the voxels of a cloud, and a right-hand side."""
    xyz, _ = _torus(case["n"], case["n"])
    keys = torch.unique(_pack(_corners(xyz, case["voxel"], 1)))
    alpha = np.random.default_rng(int(seed)).uniform(0.3, 0.7)
    c = np.array([1, 26, 66, 26, 1]) / 30.0            # products of the quadratic B-spline and of its derivative
    g = np.array([-4, -8, 24, -8, -4]) / 6.0
    cols, vals, n = [], [], keys.numel()
    for k in range(125):
        x, y, z = k // 25, k // 5 % 5, k % 5
        want = keys + (((x - 2) << 42) + ((y - 2) << 21) + (z - 2))
        at = torch.searchsorted(keys, want).clamp(max=n - 1)
        cols.append(torch.where(keys[at] == want, at, -1))
        vals.append(g[x] * c[y] * c[z] + c[x] * g[y] * c[z] + c[x] * c[y] * g[z] + alpha * c[x] * c[y] * c[z])
    cols = torch.stack(cols, 1)
    keep = cols >= 0
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(keep.sum(1), 0)
    vals = torch.tensor(vals, dtype=torch.float64, device=DEV).expand(n, 125)[keep].float()
    p = _unpack(keys).double() * case["voxel"]
    b = (torch.sin(p @ torch.tensor([31.0, 17.0, 23.0], dtype=torch.float64, device=DEV)) +
         0.3 * _randn(_gen(seed + 1), n)).float()
    return ptr, cols[keep].int(), vals, b


def _sdf_inputs(case, seed):
    xyz, nrm = _torus(case["n"], seed)
    g = _gen(seed + 1)
    near = torch.randint(case["n"], (case["queries"],), generator=g, device=DEV)
    q = xyz[near] + 0.02 * _randn(g, case["queries"], 3).float()
    far = _rand(g, case["queries"] // 16, 3).float() * 2 - 1
    q[:far.shape[0]] = far
    return q.contiguous(), xyz, nrm


def _field_inputs(case, seed):
    xyz, nrm = _torus(case["n"], seed)
    md = _min_density(xyz, case["voxel"], case["depth"], case["share"])
    g = _gen(seed + 1)
    near = torch.randint(case["n"], (case["queries"],), generator=g, device=DEV)
    pos = (xyz[near].double() + case["voxel"] * _randn(g, case["queries"], 3)).float().contiguous()
    return xyz, nrm, md, pos


# ----------------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind, s = case["kind"], dict(case)
    if kind == "reconstruct":
        s["xyz"], s["nrm"] = _cloud_inputs(case, seed)
        s["md"] = _min_density(s["xyz"], case["voxel"], case["depth"], case["share"])
    elif kind == "field":
        from jspsr.core.pipeline import Reconstruction
        xyz, nrm, md, s["pos"] = _field_inputs(case, seed)
        rec = Reconstruction(xyz, nrm, case["voxel"], case["depth"], md).build_tree()
        for lv in rec.levels:
            lv.x32 = _coefficients(lv.coords, lv.stride, case["voxel"], seed)
        s["rec"] = rec
    elif kind == "mesh":
        xyz, _ = _torus(case["n"], case["n"])
        md = _min_density(xyz, case["voxel"], case["depth"], case["share"])
        s["wave"] = torch.tensor(np.random.default_rng(int(seed)).uniform(10, 40, 2), dtype=torch.float32, device=DEV)
        s["cells"] = _leaf_cells(xyz, case["voxel"], case["depth"], md)
        while len(s["cells"][-1]) == 0:
            s["cells"].pop()
    elif kind == "solve":
        s["ptr"], s["cols"], s["vals"], s["b"] = _system(case, seed)
    elif kind == "learned":
        from jspsr import synthetic
        from jspsr.core.learned import hermite_basis
        s["basis"], s["problems"] = hermite_basis().to(DEV), []
        for i in range(case["shapes"]):
            t = [torch.from_numpy(a).to(DEV) for a in synthetic.learned_problem(case["n"], case["queries"], seed=i)]
            g = _gen(int(seed) * 64 + i)
            t[1] = _noisy(t[1], g)
            t[2] = (t[2] + 0.002 * _randn(g, *t[2].shape).float()).contiguous()
            md = _min_density(t[0], case["voxel"], case["depth"], 0.5)
            feats = _steps(s, [(*t, md)])[0].init_features(0.1, seed=int(seed) * 64 + i)
            s["problems"].append((*t, md, feats))
    elif kind == "conv":
        s["n_in"], s["n_out"], s["maps"], s["sizes"], s["x"], s["w"], s["gy"] = _conv_inputs(case, seed)
        if case["train"]:
            s["x"].requires_grad_(True)
            s["w"].requires_grad_(True)
    else:
        s["q"], s["xyz"], s["nrm"] = _sdf_inputs(case, seed)
    return s


def _steps(s, problems):
    from jspsr.core.learned import LearnedStep
    return [LearnedStep(*p[:4], voxel_size=s["voxel"], depth=s["depth"], min_density=p[4], basis=s["basis"]).build()
            for p in problems]


def _torus_field(pos, wave, R=0.31, r=0.13):
    """A field whose zero set is the torus: its distance times a positive wave."""
    d = r - torch.sqrt((torch.sqrt(pos[:, 0] ** 2 + pos[:, 1] ** 2) - R) ** 2 + pos[:, 2] ** 2)
    return d * (1.0 + 0.5 * torch.sin(wave[0] * pos[:, 0] + wave[1]))


# ----------------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "reconstruct":
        import jspsr
        _, _, rec = jspsr.reconstruct(s["xyz"], s["nrm"], s["voxel"], depth=s["depth"], min_density=s["md"],
                                      return_reconstruction=True)
        return {"solutions": [lv.x32 for lv in rec.levels], "values": rec.mesh_info["values"],
                "positions": rec.mesh_info["positions"]}
    if kind == "field":
        return s["rec"].chi_raw(s["pos"]), s["rec"].chi_raw(s["pos"], grad=True)
    if kind == "mesh":
        from types import SimpleNamespace
        from jspsr.core.pipeline import DualMesher
        m = DualMesher()
        m.levels = [SimpleNamespace(stride=2 ** d) for d in range(len(s["cells"]))]
        m.vs, m.dev = s["voxel"], s["cells"][0].device
        return m.mesh_from_leaves(dict(enumerate(s["cells"])), len(s["cells"]), 2, lambda p: _torus_field(p, s["wave"]))
    if kind == "solve":
        from jspsr import ext
        return ext.sparse_solve.solve_cusparse(s["ptr"], s["cols"], s["vals"], s["b"], 1e-12)
    if kind == "learned":
        from jspsr.core.learned import LearnedBatch
        batch = LearnedBatch(_steps(s, s["problems"]))
        normals = [p[1].clone().requires_grad_(True) for p in s["problems"]]
        feats = [{d: f.clone().requires_grad_(True) for d, f in p[5].items()} for p in s["problems"]]
        total, losses, chi = batch.forward(normals, feats)
        total.backward()
        return {"loss": torch.stack([v.detach() for v in losses]), "chi": [c.detach() for c in chi],
                "normals": [n.grad for n in normals], "features": [[f.grad for f in fs.values()] for fs in feats]}
    if kind == "conv":
        from jspsr.sparse_conv import sparse_conv
        if not s["train"]:
            with torch.no_grad():
                return sparse_conv(s["x"], s["w"], s["maps"], s["sizes"], (s["n_in"], s["n_out"]))
        y = sparse_conv(s["x"], s["w"], s["maps"], s["sizes"], (s["n_in"], s["n_out"]))
        gx, gw = torch.autograd.grad(y, [s["x"], s["w"]], s["gy"])
        return y.detach(), gx, gw
    from jspsr import sdfgen
    if s["want"] == "knn":
        return sdfgen.knn(s["q"], s["xyz"], s["k"])
    return sdfgen.sdf_from_points(s["q"], s["xyz"], s["nrm"], s["k"], 0.02)


# ----------------------------------------------------------------------------- work
def _voxels(n, voxel):
    """About how many voxels a cloud of n points on these surfaces occupies."""
    return min(5.0 * n, 5.0 / voxel ** 2)


def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "reconstruct":
        # points and normals in; solutions, samples, vertices and triangles out; some 40 products with
        # 60 entries a row
        v = _voxels(n, case["voxel"])
        return {"bytes": 24.0 * n + 5.0 * v + 18.0 * v * 4 + 3.0 * v * 12 + 6.0 * v * 24, "flops": 40 * 120.0 * v}
    if kind == "field":
        v, q = _voxels(n, case["voxel"]), case["queries"]
        return {"bytes": 2 * 12.0 * q + 16.0 * q + 2 * 6.0 * v, "flops": case["depth"] * q * (27 * 2.0 + 27 * 6.0)}
    if kind == "mesh":
        v = _voxels(n, case["voxel"])
        return {"bytes": 2.3 * v * 12 + 3.0 * v * 12 + 6.0 * v * 24, "flops": 18 * 12.0 * v}
    if kind == "solve":
        v = _voxels(n, case["voxel"])
        return {"bytes": 60.0 * v * 8 + 8 * v, "flops": 120.0 * v * 80}
    if kind == "learned":
        v = _voxels(n, case["voxel"]) * case["shapes"]
        return {"bytes": 2 * (24.0 * n + 16.0 * case["queries"]) * case["shapes"] + 2 * 18 * 4.0 * v,
                "flops": 3 * 60.0 * v * 6 * 200 + 2 * 120.0 * v * 80}
    if kind == "conv":
        v, size = _voxels(n, case["voxel"]), 4 if case["dtype"] == "f32" else 2
        K, passes = case["kernel"] ** 3, 3 if case["train"] else 1
        pairs = v * (17 if case["kernel"] == 3 else 1)
        flops = 2.0 * pairs * case["cin"] * case["cout"]
        return {"bytes": passes * (size * (v * (case["cin"] + case["cout"]) + K * case["cin"] * case["cout"]) +
                                   8.0 * pairs), "flops": passes * flops}
    q = case["queries"]
    return {"bytes": 24.0 * n + 12.0 * q + (8.0 * case["k"] * q if case["want"] == "knn" else 4.0 * q),
            "flops": 16 * 9 * 8.0 * q}


# ----------------------------------------------------------------------------- exact
def _exact_field(case, seed):
    xyz, _, md, pos = _field_inputs(case, seed)
    q = pos.double() / case["voxel"]
    val = torch.zeros(len(q), dtype=torch.float64, device=DEV)
    grad = torch.zeros(len(q), 3, dtype=torch.float64, device=DEV)
    for d, keys in enumerate(_levels(xyz, case["voxel"], case["depth"], md)):
        s = 2 ** d
        x = _coefficients(_unpack(keys), s, case["voxel"], seed).double()
        cell = (q / s).floor() * s
        for k in range(27):
            c = cell + s * torch.tensor([k // 9 - 1, k // 3 % 3 - 1, k % 3 - 1], dtype=torch.float64, device=DEV)
            want = _pack(c.long())
            at = torch.searchsorted(keys, want).clamp(max=keys.numel() - 1)
            xv = torch.where(keys[at] == want, x[at], torch.zeros((), dtype=torch.float64, device=DEV))
            rel = (q - c) / s - 0.5
            b, db = _bspline(rel), _dbspline(rel) / s
            val += b.prod(1) * xv
            grad += torch.stack([db[:, 0] * b[:, 1] * b[:, 2], b[:, 0] * db[:, 1] * b[:, 2],
                                 b[:, 0] * b[:, 1] * db[:, 2]], 1) * xv[:, None]
    return val, grad


def _exact_solve(case, seed):
    ptr, cols, vals, b = _system(case, seed)
    a = torch.sparse_csr_tensor(ptr, cols.long(), vals.double(), (len(b), len(b)))
    rows = torch.repeat_interleave(torch.arange(len(b), device=DEV), ptr[1:] - ptr[:-1])
    dinv = 1 / vals.double()[cols.long() == rows]
    b = b.double()
    x, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(3000):
        ap = a @ p
        alpha = rz / torch.dot(p, ap)
        x += alpha * p
        r -= alpha * ap
        if float(r.norm() / b.norm()) < 1e-14:
            break
        z = dinv * r
        new = torch.dot(r, z)
        p, rz = z + (new / rz) * p, new
    return x


def _exact_conv(case, seed):
    n_in, n_out, maps, sizes, x, w, gy = _conv_inputs(case, seed)
    x, w, gy, at = x.double(), w.double(), gy.double(), 0
    y = torch.zeros(n_out, case["cout"], dtype=torch.float64, device=DEV)
    gx, gw = torch.zeros_like(x), torch.zeros_like(w)
    for k, m in enumerate(sizes.tolist()):
        i, o = maps[at:at + m, 0].long(), maps[at:at + m, 1].long()
        at += m
        y.index_add_(0, o, x[i] @ w[k])
        if case["train"]:
            gx.index_add_(0, i, gy[o] @ w[k].T)
            gw[k] = x[i].T @ gy[o]
    return (y, gx, gw) if case["train"] else y


def _exact_sdf(case, seed):
    q, xyz, nrm = (t.double() for t in _sdf_inputs(case, seed))
    k, sdf, dist = case["k"], [], []
    step = max(16, int(2.5e8 / len(xyz)))
    for c in q.split(step):
        d2 = sum((c[:, None, a] - xyz[None, :, a]) ** 2 for a in range(3))
        near, at = torch.topk(d2, k, dim=1, largest=False, sorted=True)
        dist.append(near)
        ray = c[:, None] - xyz[at]
        dot = (nrm[at] * ray).sum(-1)
        first = near[:, 0].sqrt()
        mag = torch.where(first < 0.02, dot[:, 0].abs(), first)
        sdf.append(torch.where((dot > 0).sum(1) <= k // 2, -mag, mag))
    return (None, torch.cat(dist)) if case["want"] == "knn" else torch.cat(sdf)


def exact(case, seed):
    if case["kind"] == "field":
        return _exact_field(case, seed)
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "conv":
        return _exact_conv(case, seed)
    if case["kind"] == "sdf":
        return _exact_sdf(case, seed)
    return None          # whole reconstructions and training steps: no short 64-bit form; meshes: whole numbers decide
