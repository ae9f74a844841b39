"""The workloads by which this package's speed is judged, each a call through its public entry points.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges, ``prepare`` builds what a program holds
before the call (on the GPU, from the seed alone), ``run`` is one pass, ``work`` what a pass cannot do without and
``exact`` the same results in float64 from plain torch.  Sizes are those of the benchmark, the tests and the
configurations they stand for: the 10,000-Gaussian plain scene, the 3M-Gaussian scene seen from inside, the
45,304-face mesh with six Gaussians per face, FlexiCubes grids of 64 to 250 cells a side.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dmgs_gb300 import GaussianRasterizationSettings, GaussianRasterizer
from dmgs_gb300.batched import BatchedRasterizer
from dmgs_gb300.binding import barycentric_table, bind_faces, bind_faces_scale_rot
from dmgs_gb300.camera import make_view
from dmgs_gb300.flexicubes import FlexiCubes
from dmgs_gb300.loss import l1_ssim_loss
from dmgs_gb300.scenes import hemisphere_views, large_scene_tensors, random_inside_view
from dmgs_gb300.shcolor import sh_colors
from dmgs_gb300.texture import MLPTexture3D

DEV = "cuda"
MIXED = [(400, 400), (800, 800), (1237, 822), (1600, 900)]


def listed():
    return [
        # the plain rasteriser on a toy scene, one training view: latency and launches
        dict(name="splat_train_10k", kind="splat", scene="uniform", P=10_000, width=256, height=256, degree=3, grad=True),
        # stage-1 / stage-3 training of a large captured scene, one view per call
        dict(name="splat_train_3M", kind="splat", scene="inside", P=3_000_000, width=1237, height=822, degree=3, grad=True),
        # rendering test views of a finished scene: forward alone
        dict(name="splat_render_1M", kind="splat", scene="inside", P=1_000_000, width=1600, height=900, degree=3, grad=False),
        # the stage-2 rasteriser call: mesh-bound Gaussians with given covariances and colours
        dict(name="splat_mesh_272k", kind="splat", scene="mesh", P=271_824, width=800, height=800, degree=3, grad=True),
        # the headline: 16 views of the large scene per step, forward and backward, replayed as a graph
        dict(name="batch16_train_3M", kind="batch", P=3_000_000, views=16, width=1237, height=822, graph=True),
        # a batch of views of different resolutions, with each view's screen-space gradients, without a graph
        dict(name="batch4_mixed_500k", kind="batch", P=500_000, views=4, width=0, height=0, graph=False),
        # SH features of the mesh-bound Gaussians from the hash-grid texture, with its gradients
        dict(name="texture_train_272k", kind="texture", points=271_824, channels=48, grad=True),
        # extraction of the stage-2 mesh, every step, with the gradients of field, grid and weights
        dict(name="flexicubes_128", kind="flexicubes", rx=128, ry=128, rz=128),
        # stage-2 binding of the 64^3 mesh's faces
        dict(name="bind_cov_45k", kind="bind", form=2, faces=45_304, per_face=6),
        # stage-3 binding of a mesh of the finest grids
        dict(name="bind_scale_rot_700k", kind="bind", form=3, faces=700_000, per_face=6),
        # sigmoid(SH) colours of the Gaussians of a fine mesh, with gradients
        dict(name="sh_colors_1M", kind="shcolor", P=1_000_000, degree=3),
        # the photometric loss of one training view
        dict(name="l1_ssim_1237x822", kind="loss", width=1237, height=822),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["splat", "splat", "splat", "batch", "texture", "flexicubes", "bind", "shcolor", "loss"])
    w, h = rng.choice(MIXED + [(_log(rng, 200, 1600), _log(rng, 200, 1000))] * 3)
    if kind == "splat":
        scene = rng.choice(["uniform", "inside", "inside", "mesh"])
        P = _log(rng, 10_000, {"uniform": 300_000, "inside": 3_000_000, "mesh": 1_500_000}[scene])
        return dict(kind=kind, scene=scene, P=P, width=w, height=h, degree=rng.choice([0, 1, 2, 3, 3, 3]),
                    grad=rng.random() < 0.7)
    if kind == "batch":
        mixed = rng.random() < 0.5
        return dict(kind=kind, P=_log(rng, 100_000, 2_000_000), views=rng.randint(2, 16), width=0 if mixed else w,
                    height=0 if mixed else h, graph=rng.random() < 0.5)
    if kind == "texture":
        return dict(kind=kind, points=_log(rng, 20_000, 1_000_000), channels=rng.choice([3, 12, 27, 48, 48]),
                    grad=rng.random() < 0.7)
    if kind == "flexicubes":
        return dict(kind=kind, rx=_log(rng, 48, 250), ry=_log(rng, 48, 250), rz=_log(rng, 48, 250))
    if kind == "bind":
        return dict(kind=kind, form=rng.choice([2, 3]), faces=_log(rng, 20_000, 1_000_000), per_face=rng.choice([1, 3, 6, 6]))
    if kind == "shcolor":
        return dict(kind=kind, P=_log(rng, 50_000, 4_000_000), degree=rng.choice([0, 1, 2, 3, 3]))
    return dict(kind=kind, width=w, height=h)


# ---- inputs ---------------------------------------------------------------------------------------------------

class _State:
    """What a program keeps between calls; `leaves` are the tensors it takes gradients of."""

    def __init__(self, case, seed):
        self.case = case
        self.rng = np.random.default_rng(seed)
        self.gen = torch.Generator(device=DEV).manual_seed(int(seed))
        self.leaves = {}

    def randn(self, *shape):
        return torch.randn(*shape, device=DEV, generator=self.gen)

    def rand(self, *shape):
        return torch.rand(*shape, device=DEV, generator=self.gen)

    def leaf(self, name, t):
        self.leaves[name] = t.contiguous().requires_grad_(True)
        return self.leaves[name]


def _grid_mesh(S, faces):
    """A closed wavy torus of exactly `faces` triangles (the last row of quads may be cut), vertices and faces in
    scan order as an extraction leaves them."""
    nv = max(3, int(math.sqrt(faces / 6)))
    nu = -(-faces // (2 * nv))
    u = torch.arange(nu, device=DEV).view(-1, 1) * (2 * math.pi / nu)
    v = torch.arange(nv, device=DEV).view(1, -1) * (2 * math.pi / nv)
    k = [int(x) for x in S.rng.integers(2, 7, 4)]
    r = 0.3 + 0.05 * torch.sin(k[0] * u) * torch.cos(k[1] * v) + 0.02 * torch.cos(k[2] * u + k[3] * v)
    R = 0.7 + r * torch.cos(v)
    p = torch.stack([R * torch.cos(u), r * torch.sin(v).expand_as(r), R * torch.sin(u)], -1).reshape(-1, 3)
    p = p + 0.1 / nv * (S.rand(*p.shape) - 0.5)
    i, j = torch.meshgrid(torch.arange(nu, device=DEV), torch.arange(nv, device=DEV), indexing="ij")
    a, b = i * nv + j, i * nv + (j + 1) % nv
    c, d = (i + 1) % nu * nv + j, (i + 1) % nu * nv + (j + 1) % nv
    f = torch.stack([torch.stack([a, c, b], -1), torch.stack([b, c, d], -1)], 2).reshape(-1, 3)
    return p.contiguous(), f[:faces].contiguous()


def _surface_points(S, n):
    """n Gaussian centres on a mesh, six per face in face order, and the triangles' edge length."""
    F = -(-n // 6)
    verts, faces = _grid_mesh(S, F)
    bc, _ = barycentric_table(6, DEV)
    tri = verts[faces]
    return (bc @ tri).reshape(-1, 3)[:n].contiguous(), tri, float((tri[:, 1] - tri[:, 0]).norm(dim=1).mean())


def _settings(view, degree, bg):
    t = lambda a: torch.tensor(np.asarray(a, np.float32), device=DEV)  # noqa: E731
    return GaussianRasterizationSettings(
        image_height=view.height, image_width=view.width, tanfovx=view.tanfovx, tanfovy=view.tanfovy, bg=bg,
        scale_modifier=1.0, viewmatrix=t(view.viewmatrix), projmatrix=t(view.projmatrix), sh_degree=degree,
        campos=t(view.campos), prefiltered=False, debug=False)


def _inside_scene(S, P, sizes):
    """The large captured scene and one camera inside it per image size.  Gaussians closer than one unit to a camera
    are moved out to that distance, as a capture has free space around its cameras, and their scales are kept within
    e^-6 and e^-2.5, as training splits the large ones and prunes the rest."""
    g = large_scene_tensors(P, int(S.rng.integers(1 << 30)), DEV)
    g["scales"] = g["scales"].clamp(min=math.exp(-6.0), max=math.exp(-2.5))
    views = [random_inside_view(S.rng, w, h) for w, h in sizes]
    for v in views:
        d = g["means3D"] - torch.tensor(v.campos, device=DEV)
        r = d.norm(dim=1, keepdim=True)
        g["means3D"] = torch.where(r < 1.0, g["means3D"] + d * (1.0 / r - 1.0), g["means3D"])
    return g, views


def _prepare_splat(S, c):
    P, w, h = c["P"], c["width"], c["height"]
    if c["scene"] == "inside":
        g, (view,) = _inside_scene(S, P, [(w, h)])
    elif c["scene"] == "uniform":
        q, sh = S.randn(P, 4), 0.05 * S.randn(P, 16, 3)
        sh[:, 0] = 0.5 + 0.2 * S.randn(P, 3)
        # scales shrink with the density beyond 10,000 Gaussians, as a densified scene's do
        g = dict(means3D=2 * S.rand(P, 3) - 1, scales=torch.exp(-5 + 2 * S.rand(P, 3)) * (1e4 / P) ** (1 / 3),
                 rotations=q / q.norm(dim=1, keepdim=True), opacities=torch.sigmoid(S.randn(P, 1)), shs=sh)
        view = make_view(4.0 * np.array([0.47, 0.34, 0.81]), (0.0, 0.0, 0.0), w, h, fovx_deg=50.0)
    else:
        xyz, _, edge = _surface_points(S, P)
        L = S.randn(P, 3, 3) * (0.15 * edge)
        L[:, 2] *= 0.05
        A = torch.linalg.qr(S.randn(-(-P // 6), 3, 3))[0].repeat_interleave(6, 0)[:P] @ L
        C = A @ A.transpose(1, 2)
        cov = torch.stack([C[:, 0, 0], C[:, 0, 1], C[:, 0, 2], C[:, 1, 1], C[:, 1, 2], C[:, 2, 2]], 1)
        g = dict(means3D=xyz, cov3D_precomp=cov, colors_precomp=S.rand(P, 3), opacities=torch.full((P, 1), 0.9999, device=DEV))
        view = hemisphere_views(1, w, h, seed=int(S.rng.integers(1 << 30)))[0]
    S.g = {k: S.leaf(k, v) if c["grad"] else v.contiguous() for k, v in g.items()}
    S.means2D = torch.zeros(P, 3, device=DEV)
    if c["grad"]:
        S.leaf("means2D", S.means2D)
        S.dimage = S.randn(3, h, w) / (3 * h * w)
    S.view = view
    S.raster = GaussianRasterizer(_settings(view, c["degree"], S.rand(3)))


def _prepare_batch(S, c):
    S.g, S.view = _inside_scene(S, c["P"], [MIXED[k % 4] if not c["width"] else (c["width"], c["height"])
                                            for k in range(c["views"])])
    S.br = BatchedRasterizer([_settings(v, 3, torch.zeros(3, device=DEV)) for v in S.view], S.g,
                             means2D_grads=not c["graph"], densify_stats=c["graph"])
    for d in S.br.dL_dout:
        d.copy_(S.randn(*d.shape) / d.numel())
    if c["graph"]:
        S.br.capture()


def _prepare_texture(S, c):
    xyz, _, _ = _surface_points(S, c["points"])
    torch.manual_seed(int(S.rng.integers(1 << 30)))
    S.aabb = torch.stack([xyz.min(0).values, xyz.max(0).values]) * 1.1
    S.tex = MLPTexture3D(S.aabb, channels=c["channels"], device=DEV)
    with torch.no_grad():  # a table as training leaves it: features of order one
        S.tex.encoder.params.copy_(0.5 * S.randn(S.tex.encoder.params.numel()))
    S.xyz = xyz
    S.params = [S.tex.encoder.params] + S.tex.net.weights()
    if c["grad"]:
        S.xyz = S.leaf("xyz", xyz)
        for name, p in zip(("table", "W1", "W2", "W3"), S.params):
            S.leaves[name] = p
        S.dout = S.randn(c["points"], c["channels"])


def _prepare_flexicubes(S, c):
    S.res = (c["rx"], c["ry"], c["rz"])
    S.fc = FlexiCubes(device=DEV)
    S.grid, S.cubes = S.fc.construct_voxel_grid_v2(S.res, [-1.0] * 3, [1.0] * 3)
    cell = 2.0 / max(S.res)
    p = S.grid
    s = p.norm(dim=1) - 0.7 + 0.08 * torch.sin(3.1 * p[:, 0]) * torch.cos(2.3 * p[:, 1]) + 0.05 * torch.sin(2.7 * p[:, 2])
    # the field's values vary with the seed, its signs do not: every seed's mesh has the same faces
    S.s = S.leaf("s", (s + 3e-4) * (0.8 + 0.4 * S.rand(s.shape[0])))
    S.x = S.leaf("x", p + 0.2 * cell * (S.rand(*p.shape) - 0.5))
    S.w = S.leaf("weights", 1.0 + 0.1 * S.randn(S.cubes.shape[0], 21))
    v, _, L, _ = _extract(S)
    S.dv, S.dL = S.randn(*v.shape), S.rand(*L.shape) / L.shape[0]


def _extract(S):
    w = S.w
    return S.fc(S.x, S.s, S.cubes, S.res, w[:, :12], w[:, 12:20], w[:, 20], training=True)


def _prepare_bind(S, c):
    verts, S.faces = _grid_mesh(S, c["faces"])
    S.verts = S.leaf("verts", verts)
    S.bc, S.rad = barycentric_table(c["per_face"], DEV)
    n = c["faces"] * c["per_face"]
    if c["form"] == 2:
        S.scale = S.leaf("scale_factor", torch.full((1,), math.atanh(0.5), device=DEV) + 0.1 * S.rand(1))
        S.grads = [S.randn(n, 3), S.randn(n, 6)]
    else:
        S.s2 = S.leaf("scaling2d", math.log(1.0 / math.sqrt(c["faces"])) + 0.3 * S.randn(n, 2))
        S.r2 = S.leaf("rotation2d", S.randn(n, 2))
        S.grads = [S.randn(n, 3), S.randn(n, 3), S.randn(n, 4)]


def _prepare_shcolor(S, c):
    P, K = c["P"], (c["degree"] + 1) ** 2
    xyz, _, _ = _surface_points(S, P)
    sh = 0.2 * S.randn(P, 3, K)
    sh[:, :, 0] += 0.5
    S.sh, S.xyz = S.leaf("sh", sh), S.leaf("xyz", xyz)
    S.campos = torch.tensor(hemisphere_views(1, 8, 8, seed=int(S.rng.integers(1 << 30)))[0].campos, device=DEV)
    S.dcol = S.randn(P, 3)


def _prepare_loss(S, c):
    shape = (3, c["height"], c["width"])
    y = torch.nn.functional.interpolate(S.rand(1, 3, 2 + shape[1] // 8, 2 + shape[2] // 8), size=shape[1:], mode="bilinear")[0]
    S.target = y.contiguous()
    S.image = S.leaf("image", (y + 0.05 * S.randn(*shape)).clamp(0, 1))


def prepare(case, seed):
    S = _State(case, seed)
    globals()["_prepare_" + case["kind"]](S, case)
    return S


# ---- one pass -------------------------------------------------------------------------------------------------

def _grads(S, outs, douts):
    return dict(zip(S.leaves, torch.autograd.grad(outs, list(S.leaves.values()), douts)))


def run(state):
    S, c = state, state.case
    kind = c["kind"]
    if kind == "splat":
        g = S.g
        with torch.set_grad_enabled(c["grad"]):
            image, radii = S.raster(means3D=g["means3D"], means2D=S.means2D, opacities=g["opacities"], shs=g.get("shs"),
                                    colors_precomp=g.get("colors_precomp"), scales=g.get("scales"),
                                    rotations=g.get("rotations"), cov3D_precomp=g.get("cov3D_precomp"))
        out = dict(image=image.detach(), radii=radii)
        if c["grad"]:
            out["grad"] = _grads(S, [image], [S.dimage])
        return out
    if kind == "batch":
        S.br.reset_densify_stats()
        S.br.step()
        out = dict(images=S.br.images, radii=S.br.radii, grad={k: v for k, v in S.br.grads.items() if v is not None})
        if c["graph"]:
            out.update(densify=[S.br.densify_accum, S.br.densify_count])
        else:
            out.update(means2D=S.br.means2D_grads)
        return out
    if kind == "texture":
        if not c["grad"]:
            with torch.no_grad():
                return dict(features=S.tex.sample_noact(S.xyz))
        f = S.tex.sample_noact(S.xyz)
        return dict(features=f.detach(), grad=_grads(S, [f], [S.dout]))
    if kind == "flexicubes":
        v, f, L, e = _extract(S)
        return dict(vertices=v.detach(), faces=f, L_dev=L.detach(), edges=e, grad=_grads(S, [v, L], [S.dv, S.dL]))
    if kind == "bind":
        if c["form"] == 2:
            xyz, cov, L = bind_faces(S.verts, S.faces, S.bc, S.scale, S.rad, 1.0)
            outs, more = [xyz, cov], [L]
        else:
            outs, more = list(bind_faces_scale_rot(S.verts, S.faces, S.bc, S.s2, S.r2, 1e-6)), []
        return dict(outs=[o.detach() for o in outs] + more, grad=_grads(S, outs, S.grads))
    if kind == "shcolor":
        col = sh_colors(c["degree"], S.sh, S.xyz, S.campos)
        return dict(colors=col.detach(), grad=_grads(S, [col], [S.dcol]))
    loss = l1_ssim_loss(S.image, S.target)
    return dict(loss=loss.detach(), grad=torch.autograd.grad(loss, [S.image])[0])


# ---- what a pass cannot do without ------------------------------------------------------------------------------

def work(case):
    """Inputs read once, outputs written once.  Flops: of the arithmetic per item where it is fixed; the blends' grows
    with the scene and is left out."""
    c, kind = case, case["kind"]
    if kind == "splat":
        per = 12 + 4 + (24 + 12 if c["scene"] == "mesh" else 12 + 16 + 192)
        image = 12 * c["width"] * c["height"]
        b = c["P"] * (per + 4) + image
        return dict(bytes=b + (c["P"] * (per + 12) + image if c["grad"] else 0), flops=0)
    if kind == "batch":
        sizes = [MIXED[k % 4] if not c["width"] else (c["width"], c["height"]) for k in range(c["views"])]
        image = sum(12 * w * h for w, h in sizes)
        return dict(bytes=c["P"] * (2 * 236 + c["views"] * (4 if c["graph"] else 16) + (8 if c["graph"] else 0)) + 2 * image, flops=0)
    if kind == "texture":
        n, C = c["points"], c["channels"]
        mlp = 2 * n * (32 * 32 * 2 + 32 * C)
        table = 8 * min(6_299_960, 128 * n)
        if not c["grad"]:
            return dict(bytes=n * (12 + 4 * C) + table, flops=mlp)
        return dict(bytes=n * (24 + 8 * C) + table + 8 * 6_299_960, flops=3 * mlp)
    if kind == "flexicubes":
        n = c["rx"] * c["ry"] * c["rz"]
        surf = 4 * max(c["rx"], c["ry"], c["rz"]) ** 2
        return dict(bytes=n * (4 + 12 + 4 + 84) + surf * (84 * 2 + 12 * 8 + 300), flops=0)
    if kind == "bind":
        F, n = c["faces"], c["faces"] * c["per_face"]
        per = 12 + 24 if c["form"] == 2 else 12 + 12 + 16
        extra = 36 * F if c["form"] == 2 else 16 * n * 2
        return dict(bytes=F * (24 + 6) + n * per * 2 + extra + 12 * F // 2, flops=0)
    if kind == "shcolor":
        K = (c["degree"] + 1) ** 2
        return dict(bytes=c["P"] * (12 * K * 2 + 12 * 4), flops=c["P"] * 20 * K)
    n = 3 * c["width"] * c["height"]
    return dict(bytes=12 * n, flops=n * 2 * 11 * 2 * 8)


# ---- the same results in float64 ----------------------------------------------------------------------------------

_C0, _C1 = 0.28209479177387814, 0.4886025119029199
_C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
_C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
       1.445305721320277, -0.5900435899266435)


def _sh_basis(degree, d):
    """The real SH basis [P, (degree + 1)^2] at unit directions d [P, 3]."""
    x, y, z = d.unbind(1)
    b = [torch.full_like(x, _C0)]
    if degree > 0:
        b += [-_C1 * y, _C1 * z, -_C1 * x]
    if degree > 1:
        xx, yy, zz = x * x, y * y, z * z
        b += [_C2[0] * x * y, _C2[1] * y * z, _C2[2] * (2 * zz - xx - yy), _C2[3] * x * z, _C2[4] * (xx - yy)]
    if degree > 2:
        b += [_C3[0] * y * (3 * xx - yy), _C3[1] * x * y * z, _C3[2] * y * (4 * zz - xx - yy),
              _C3[3] * z * (2 * zz - 3 * xx - 3 * yy), _C3[4] * x * (4 * zz - xx - yy), _C3[5] * z * (xx - yy),
              _C3[6] * x * (xx - 3 * yy)]
    return torch.stack(b, 1)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _double(t):
    return None if t is None else t.detach().double().requires_grad_(True)


def _quat_matrix(q):
    r, x, y, z = q.unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y),
                        2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x),
                        2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)


def _project(g, ndc_shift, rs, degree):
    """Radii (0: culled) and, per Gaussian, pixel position, conic, opacity, colour and depth, differentiable; the
    conventions of the published rasteriser's adjoint (the field-of-view clamp holds its value constant)."""
    W, H = rs.image_width, rs.image_height
    V, Pm, cam = rs.viewmatrix.double(), rs.projmatrix.double(), rs.campos.double()
    m = g["means3D"]
    t = m @ V[:3, :3] + V[3, :3]
    hom = m @ Pm[:3] + Pm[3]
    ndc = hom[:, :2] / (hom[:, 3:] + 1e-7) + ndc_shift[:, :2]
    pix = ((ndc + 1) * torch.tensor([W, H], device=DEV).double() - 1) / 2
    front = t[:, 2] > 0.2
    z = torch.where(front, t[:, 2], torch.ones_like(t[:, 2]))
    tan = torch.tensor([rs.tanfovx, rs.tanfovy], device=DEV, dtype=torch.float64)
    focal = torch.tensor([W, H], device=DEV).double() / (2 * tan)
    lim = 1.3 * tan
    ratio = t[:, :2] / z[:, None]
    inside = ratio.abs() <= lim
    txy = torch.where(inside, t[:, :2], (torch.maximum(torch.minimum(ratio, lim), -lim) * z[:, None]).detach())
    zero = torch.zeros_like(z)
    J = torch.stack([torch.stack([focal[0] / z, zero, -focal[0] * txy[:, 0] / z ** 2], 1),
                     torch.stack([zero, focal[1] / z, -focal[1] * txy[:, 1] / z ** 2], 1)], 1)
    if g.get("cov3D_precomp") is not None:
        s = g["cov3D_precomp"]
        Sigma = s[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].view(-1, 3, 3)
    else:
        M = _quat_matrix(g["rotations"]) * (rs.scale_modifier * g["scales"])[:, None, :]
        Sigma = M @ M.transpose(1, 2)
    T = J @ V[:3, :3].T
    cov = T @ Sigma @ T.transpose(1, 2)
    A, B, C = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = A * C - B * B
    ok = front & (det != 0)
    det = torch.where(det != 0, det, torch.ones_like(det))
    conic = torch.stack([C / det, -B / det, A / det], 1)
    mid = (A + C) / 2
    rad = torch.ceil(3 * torch.sqrt(mid + torch.sqrt((mid * mid - det).clamp(min=0.1)))).detach()
    grid = torch.tensor([-(-W // 16), -(-H // 16)], device=DEV)
    lo = torch.minimum(((pix.detach() - rad[:, None]) / 16).clamp(0, 1e6).long(), grid)
    hi = torch.minimum(((pix.detach() + rad[:, None] + 15) / 16).clamp(0, 1e6).long(), grid)
    ok = ok & (rad > 0) & ((hi - lo).prod(1) > 0)
    if g.get("colors_precomp") is not None:
        rgb = g["colors_precomp"]
    else:
        n = (degree + 1) ** 2
        rgb = ((_sh_basis(degree, _unit(m - cam))[:, :, None] * g["shs"][:, :n]).sum(1) + 0.5).clamp(min=0)
    feat = torch.cat([pix, conic, g["opacities"].view(-1, 1), rgb], 1)
    return torch.where(ok, rad, zero), feat, t[:, 2].detach(), lo, hi, ok


def _exact_view(g, shift, rs, degree, dimage):
    """Image, radii and, with dimage, the gradients w.r.t. the tensors of g and the NDC means of one view."""
    W, H = rs.image_width, rs.image_height
    bg = rs.bg.double()
    rad, feat, depth, lo, hi, ok = _project(g, shift, rs, degree)
    F = feat.detach()
    idx = torch.nonzero(ok).squeeze(1)
    idx = idx[torch.argsort(depth[idx].float(), stable=True)]
    wd = (hi - lo)[idx]
    cnt = wd.prod(1)
    own = torch.repeat_interleave(torch.arange(idx.numel(), device=DEV), cnt)
    k = torch.arange(own.numel(), device=DEV) - (cnt.cumsum(0) - cnt)[own]
    gx = -(-W // 16)
    tile = (lo[idx][own, 1] + k // wd[own, 0]) * gx + lo[idx][own, 0] + k % wd[own, 0]
    tile, order = torch.sort(tile, stable=True)
    ids = idx[own[order]]
    ends = torch.searchsorted(tile, torch.arange(gx * -(-H // 16) + 1, device=DEV)).tolist()
    image = torch.zeros(3, H, W, device=DEV, dtype=torch.float64) + bg[:, None, None]
    dfeat = torch.zeros_like(F)
    for t in range(len(ends) - 1):
        a, b = ends[t], ends[t + 1]
        if a == b:
            continue
        y0, x0 = t // gx * 16, t % gx * 16
        y1, x1 = min(H, y0 + 16), min(W, x0 + 16)
        yy, xx = torch.meshgrid(torch.arange(y0, y1, device=DEV), torch.arange(x0, x1, device=DEV), indexing="ij")
        f = F[ids[a:b]].requires_grad_(dimage is not None)
        dx, dy = f[:, 0] - xx.reshape(-1, 1), f[:, 1] - yy.reshape(-1, 1)
        power = -0.5 * (f[:, 2] * dx * dx + f[:, 4] * dy * dy) - f[:, 3] * dx * dy
        al = f[:, 5] * torch.exp(power)
        al = al + (al.clamp(max=0.99) - al).detach()  # the cap is not differentiated
        al = torch.where((power <= 0) & (al >= 1 / 255), al, torch.zeros_like(al))
        al = torch.where(torch.cumprod(1 - al.detach(), 1) >= 1e-4, al, torch.zeros_like(al))
        T = torch.cumprod(1 - al, 1)
        Tb = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1)
        col = (al * Tb) @ f[:, 6:] + T[:, -1:] * bg
        image[:, y0:y1, x0:x1] = col.detach().T.reshape(3, y1 - y0, x1 - x0)
        if dimage is not None:
            (d,) = torch.autograd.grad(col, f, dimage[:, y0:y1, x0:x1].reshape(3, -1).T)
            dfeat.index_add_(0, ids[a:b], d)
    if dimage is None:
        return image, rad.int(), None
    return image, rad.int(), (torch.where(ok[:, None], feat, torch.zeros_like(feat)), torch.where(ok[:, None], dfeat, torch.zeros_like(dfeat)))


def _exact_splat(S, c):
    if c["width"] * c["height"] > 1_500_000:
        return None
    rs = S.raster.raster_settings
    g = {k: _double(v) for k, v in S.g.items()}
    shift = torch.zeros(c["P"], 2, device=DEV, dtype=torch.float64, requires_grad=True)
    image, _, back = _exact_view(g, shift, rs, c["degree"], S.dimage.double() if c["grad"] else None)
    out = dict(image=image, radii=None)
    if c["grad"]:
        names = list(g)
        got = torch.autograd.grad([back[0]], [g[n] for n in names] + [shift], [back[1]])
        grad = dict(zip(names, got))
        grad["means2D"] = torch.cat([got[-1], torch.zeros(c["P"], 1, device=DEV, dtype=torch.float64)], 1)
        out["grad"] = {n: grad[n] for n in S.leaves}
    return out


def _exact_batch(S, c):
    if sum(v.width * v.height for v in S.view) > 3_000_000:
        return None  # tens of seconds
    g = {k: _double(v) for k, v in S.g.items()}
    images, m2, total = [], [], None
    n2 = torch.zeros(c["P"], device=DEV, dtype=torch.float64)
    seen = torch.zeros_like(n2)
    for rs, d in zip(S.br.settings, S.br.dL_dout):
        shift = torch.zeros(c["P"], 2, device=DEV, dtype=torch.float64, requires_grad=True)
        image, rad, back = _exact_view(g, shift, rs, 3, d.double())
        got = torch.autograd.grad([back[0]], list(g.values()) + [shift], [back[1]])
        images.append(image)
        m2.append(torch.cat([got[-1], torch.zeros(c["P"], 1, device=DEV, dtype=torch.float64)], 1))
        n2, seen = n2 + got[-1].norm(dim=1), seen + (rad > 0)
        total = list(got[:-1]) if total is None else [a + b for a, b in zip(total, got)]
    out = dict(images=images, radii=[None] * len(images), grad=dict(zip(g, total)))
    out.update(dict(densify=[n2, seen]) if c["graph"] else dict(means2D=m2))
    return out


def _exact_texture(S, c):
    x = _double(S.xyz)
    table, w1, w2, w3 = (_double(p) for p in S.params)
    lo, hi = S.aabb.double()
    t = ((x - lo) / (hi - lo)).clamp(0, 1)
    log2b = float(np.float32(math.log2(float(np.float32(math.exp(math.log(256.0) / 15))))))
    enc, off = [], 0
    rows = table.view(-1, 2)
    for lvl in range(16):
        scale = float(np.float32(2.0 ** (lvl * log2b) * 16 - 1))
        res = math.ceil(scale) + 1
        size = min(-(-res ** 3 // 8) * 8, 1 << 19)
        p = t * scale + 0.5
        cell = p.detach().floor()
        f, cell, acc = p - cell, cell.long(), 0.0
        for corner in range(8):
            bit = [(corner >> d) & 1 for d in range(3)]
            w = math.prod([f[:, d] if bit[d] else 1 - f[:, d] for d in range(3)])
            q = [cell[:, d] + bit[d] for d in range(3)]
            if res ** 3 > size:
                k = q[0] ^ (q[1] * 2654435761 & 0xFFFFFFFF) ^ (q[2] * 805459861 & 0xFFFFFFFF)
            else:
                k = q[0] + q[1] * res + q[2] * res * res
            acc = acc + w[:, None] * rows[k % size + off]
        enc.append(acc)
        off += size
    f = torch.relu(torch.relu(torch.cat(enc, 1) @ w1.T) @ w2.T) @ w3.T
    if not c["grad"]:
        return dict(features=f.detach())
    g = torch.autograd.grad([f], [x, table, w1, w2, w3], [S.dout.double()])
    return dict(features=f.detach(), grad=dict(xyz=g[0], table=128 * g[1], W1=g[2], W2=g[3], W3=g[4]))


_EDGES = [(0, 1), (1, 5), (4, 5), (0, 4), (2, 3), (3, 7), (6, 7), (2, 6), (2, 0), (3, 1), (7, 5), (6, 4)]


def _dual_sets():
    """Per corner-sign case the sets of crossing edges that share a dual vertex, [256, 4, 7] padded with -1, and
    whether a face of the cube is ambiguous."""
    table, ambiguous = np.full((256, 4, 7), -1), np.zeros(256, bool)
    for case in range(256):
        occ = [(case >> n) & 1 for n in range(8)]
        group = {e: e for e, (a, b) in enumerate(_EDGES) if occ[a] != occ[b]}
        for axis in range(3):
            for side in (0, 1):
                on = [e for e in group if all((n >> axis) & 1 == side for n in _EDGES[e])]
                ambiguous[case] |= len(on) == 4
                if len(on) == 2:
                    old, new = group[on[0]], group[on[1]]
                    group = {e: new if s == old else s for e, s in group.items()}
        minority = int(sum(occ) <= 4)
        sets = [sorted(e for e in group if group[e] == s) for s in set(group.values())]
        sets.sort(key=lambda es: [min(n for e in es for n in _EDGES[e] if occ[n] == v) for v in (minority, 1 - minority)])
        for i, es in enumerate(sets[:4]):
            table[case, i, :len(es)] = es
    return torch.tensor(table, device=DEV), torch.tensor(ambiguous, device=DEV)


def _exact_flexicubes(S, c):
    x, s, w = _double(S.x), _double(S.s), _double(S.w)
    sets, ambiguous = _dual_sets()
    occ = s < 0
    n_in = occ[S.cubes].sum(1)
    sc = torch.nonzero((n_in > 0) & (n_in < 8)).squeeze(1)
    corners = S.cubes[sc]
    case = (occ[corners].long() << torch.arange(8, device=DEV)).sum(1)
    if bool(ambiguous[case].any()):
        return None  # the neighbour rule of ambiguous cubes is not restated here
    beta, alpha = torch.tanh(w[sc, :12]) * 0.99 + 1, torch.tanh(w[sc, 12:20]) * 0.99 + 1
    gamma = torch.sigmoid(w[sc, 20]) * 0.99 + 0.005
    nvd = (sets[case, :, 0] >= 0).sum(1)
    per = [torch.nonzero(nvd == n).squeeze(1) for n in range(1, 5)]  # dual vertices: by their cube's count, then cube
    cube_of = torch.cat([p.repeat_interleave(n + 1) for n, p in enumerate(per)])
    slot = torch.cat([torch.arange(n + 1, device=DEV).repeat(p.numel()) for n, p in enumerate(per)])
    edges = sets[case[cube_of], slot]
    vd_e, k = torch.nonzero(edges >= 0).unbind(1)
    edge, cube_e = edges[vd_e, k], cube_of[vd_e]
    ends = corners[cube_e[:, None], torch.tensor(_EDGES, device=DEV)[edge]]

    def crossing(w0, w1):
        return (x[ends[:, 0]] * w1[:, None] - x[ends[:, 1]] * w0[:, None]) / (w1 - w0)[:, None]
    local = torch.tensor(_EDGES, device=DEV)[edge]
    s0, s1 = s[ends[:, 0]], s[ends[:, 1]]
    u = crossing(s0 * alpha[cube_e, local[:, 0]], s1 * alpha[cube_e, local[:, 1]])
    total, bw = cube_of.numel(), beta[cube_e, edge]
    zeros = torch.zeros(total, device=DEV, dtype=torch.float64)
    vd = torch.zeros(total, 3, device=DEV, dtype=torch.float64).index_add(0, vd_e, u * bw[:, None])
    vd = vd / zeros.index_add(0, vd_e, bw)[:, None]
    dist = (crossing(s0, s1) - vd[vd_e]).norm(dim=1)
    mean = zeros.index_add(0, vd_e, dist) / zeros.index_add(0, vd_e, torch.ones_like(dist))
    L = (dist - mean[vd_e]).abs()
    # quads: the four dual vertices around each grid edge shared by four cubes, by edge, then cube
    N = x.shape[0]
    key = ends[:, 0] * N + ends[:, 1]
    order = torch.argsort(cube_e, stable=True)
    order = order[torch.argsort(key[order], stable=True)]
    _, inv, count = torch.unique_consecutive(key[order], return_inverse=True, return_counts=True)
    full = order[count[inv] == 4].view(-1, 4)
    quad, first = vd_e[full], full[:, 0]
    flip = s[ends[first, 0]] > 0
    quad = torch.cat([quad[flip][:, [0, 1, 3, 2]], quad[~flip][:, [2, 3, 1, 0]]])
    g = gamma[cube_of][quad]
    g02, g13 = (g[:, 0] * g[:, 2])[:, None], (g[:, 1] * g[:, 3])[:, None]
    q = vd[quad]
    centre = ((q[:, 0] + q[:, 2]) / 2 * g02 + (q[:, 1] + q[:, 3]) / 2 * g13) / (g02 + g13 + 1e-8)
    v = torch.cat([vd, centre])
    d = torch.autograd.grad([v, L], [s, x, w], [S.dv.double(), S.dL.double()])
    return dict(vertices=v.detach(), faces=None, L_dev=L.detach(), edges=None, grad=dict(s=d[0], x=d[1], weights=d[2]))


def _frames(v, f):
    t = v[f]
    e1, e2 = t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    x = _unit(e1)
    n = _unit(torch.linalg.cross(e1, e2))
    y = _unit(torch.linalg.cross(n, x))
    return t, e1, e2, torch.stack([x, y, n], 2)


def _exact_bind(S, c):
    v, bc, G = _double(S.verts), S.bc.double(), c["per_face"]
    t, e1, e2, R = _frames(v, S.faces)
    xyz = (bc @ t).reshape(-1, 3)
    if c["form"] == 2:
        sf = _double(S.scale)
        with torch.no_grad():
            ln = e1.norm(dim=1)
            ax, ay = (e2 * R[:, :, 0]).sum(1), (e2 * R[:, :, 1]).sum(1)
            L = torch.zeros(len(t), 3, 3, device=DEV, dtype=torch.float64)
            ey = ln * (math.sqrt(3) / 2)
            L[:, 0, 0], L[:, 0, 1], L[:, 1, 1] = ln * S.rad, (ax - ln / 2) / ey * ln * S.rad, ay / ey * ln * S.rad
            L[:, 2, 2] = float(np.float32(1e-6))
        M = R @ L * torch.tanh(sf) * 2.0
        C = M @ M.transpose(1, 2)
        cov = C.reshape(-1, 9)[:, [0, 1, 2, 4, 5, 8]].repeat_interleave(G, 0)
        outs, more = [xyz, cov], [L]
        leaves = [v, sf]
    else:
        s2, r2 = _double(S.s2), _double(S.r2)
        a, b = _unit(r2).unbind(1)
        z, o = torch.zeros_like(a), torch.ones_like(a)
        M = R.repeat_interleave(G, 0) @ torch.stack([a, -b, z, b, a, z, z, z, o], 1).view(-1, 3, 3)
        d = M.diagonal(dim1=1, dim2=2)
        # 4 q q^T, its largest diagonal entry's row normalised: the quaternion up to its sign
        tr = d.sum(1)
        sq = torch.stack([1 + tr, 1 + 2 * d[:, 0] - tr, 1 + 2 * d[:, 1] - tr, 1 + 2 * d[:, 2] - tr], 1)
        m = lambda i, j: M[:, i, j]  # noqa: E731
        rows = torch.stack([
            torch.stack([sq[:, 0], m(2, 1) - m(1, 2), m(0, 2) - m(2, 0), m(1, 0) - m(0, 1)], 1),
            torch.stack([m(2, 1) - m(1, 2), sq[:, 1], m(1, 0) + m(0, 1), m(0, 2) + m(2, 0)], 1),
            torch.stack([m(0, 2) - m(2, 0), m(1, 0) + m(0, 1), sq[:, 2], m(2, 1) + m(1, 2)], 1),
            torch.stack([m(1, 0) - m(0, 1), m(0, 2) + m(2, 0), m(2, 1) + m(1, 2), sq[:, 3]], 1)], 1)
        best = sq.argmax(1)
        # Shepperd's form: half the root of the largest, the others through it
        root = 0.5 * torch.sqrt(sq.gather(1, best[:, None]))
        row = rows[torch.arange(len(best), device=DEV), best]
        q = torch.where(torch.nn.functional.one_hot(best, 4).bool(), root.expand(-1, 4), row * (0.25 / root))
        q = _unit(q * torch.where(q[:, :1] < 0, -1.0, 1.0))
        sc = torch.cat([torch.exp(s2), torch.full_like(s2[:, :1], float(np.float32(1e-6)))], 1)
        outs, more, leaves = [xyz, sc, q], [], [v, s2, r2]
    g = torch.autograd.grad(outs, leaves, [d.double() for d in S.grads])
    return dict(outs=[o.detach() for o in outs] + more, grad=dict(zip(S.leaves, g)))


def _exact_shcolor(S, c):
    sh, x = _double(S.sh), _double(S.xyz)
    col = torch.sigmoid((sh * _sh_basis(c["degree"], _unit(x - S.campos.double()))[:, None]).sum(2))
    g = torch.autograd.grad([col], [sh, x], [S.dcol.double()])
    return dict(colors=col.detach(), grad=dict(sh=g[0], xyz=g[1]))


def _exact_loss(S, c):
    x, y = _double(S.image), S.target.double()
    k = torch.exp(-((torch.arange(11, device=DEV).double() - 5) ** 2) / (2 * 1.5 ** 2))
    k = k / k.sum()
    w = (k[:, None] * k)[None, None].expand(3, 1, 11, 11)

    def blur(a):
        return torch.nn.functional.conv2d(a[None], w, padding=5, groups=3)
    mx, my = blur(x), blur(y)
    sxx, syy, sxy = blur(x * x) - mx * mx, blur(y * y) - my * my, blur(x * y) - mx * my
    ssim = ((2 * mx * my + 1e-4) * (2 * sxy + 9e-4)) / ((mx * mx + my * my + 1e-4) * (sxx + syy + 9e-4))
    loss = 0.8 * (x - y).abs().mean() + 0.2 * (1 - ssim.mean())
    return dict(loss=loss.detach(), grad=torch.autograd.grad(loss, [x])[0])


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](prepare(case, seed), case)
