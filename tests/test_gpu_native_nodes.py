"""The native autograd nodes against the general form (the Python
torch.autograd.Function classes) on every call form: same outputs and
gradients where the native entry takes the call, the general form's results
and errors where it does not."""
import numpy as np
import pytest
import torch

import dmgs_gb300
from dmgs_gb300 import _lib
from dmgs_gb300._lib import DmgsError
from dmgs_gb300.binding import barycentric_table, bind_faces, bind_faces_scale_rot
from dmgs_gb300.flexicubes import FlexiCubes
from dmgs_gb300.loss import l1_ssim_loss
from dmgs_gb300.scenes import small_scene
from dmgs_gb300.shcolor import sh_colors
from dmgs_gb300.texture import MLPTexture3D

pytestmark = pytest.mark.gpu
D = "cuda"


def _gen(seed):
    return torch.Generator(device=D).manual_seed(seed)


def _raster(mode):
    sc = small_scene(P=700, width=70, height=50, seed=3)
    v = sc.views[0]
    rs = dmgs_gb300.GaussianRasterizationSettings(
        image_height=50, image_width=70, tanfovx=v.tanfovx, tanfovy=v.tanfovy, bg=torch.rand(3, device=D, generator=_gen(1)),
        scale_modifier=1.1, viewmatrix=torch.tensor(v.viewmatrix, device=D), projmatrix=torch.tensor(v.projmatrix, device=D),
        sh_degree=2, campos=torch.tensor(v.campos, device=D), prefiltered=False, debug=False)
    t = lambda a: torch.tensor(a, device=D)  # noqa: E731
    g = dict(means3D=t(sc.means3D), opacities=t(sc.opacities), means2D=torch.zeros(700, 3, device=D))
    if "cov" in mode:
        A = 0.03 * torch.randn(700, 3, 3, device=D, generator=_gen(2))
        C = A @ A.transpose(1, 2)
        g["cov3D_precomp"] = torch.stack([C[:, 0, 0], C[:, 0, 1], C[:, 0, 2], C[:, 1, 1], C[:, 1, 2], C[:, 2, 2]], 1)
    else:
        g.update(scales=t(sc.scales), rotations=t(sc.rotations))
    if "colors" in mode:
        g["colors_precomp"] = torch.rand(700, 3, device=D, generator=_gen(4))
    else:
        g["shs"] = t(sc.shs)
    return g, lambda **k: dmgs_gb300.GaussianRasterizer(rs)(**k)


def _mesh(F=200, V=90):
    g = _gen(5)
    faces = torch.stack([torch.randperm(V, device=D, generator=g)[:3] for _ in range(F)])
    return torch.randn(V, 3, device=D, generator=g), faces


def _ops():
    for mode in ("sh", "colors", "cov", "cov-colors"):
        yield "raster-" + mode, lambda mode=mode: _raster(mode)

    def loss():
        x = torch.rand(3, 40, 37, device=D, generator=_gen(6))
        y = torch.rand(3, 40, 37, device=D, generator=_gen(7))
        return dict(image=x), lambda image: (l1_ssim_loss(image, y),)
    yield "loss", loss

    def sh():
        cam = torch.tensor([0.1, 3.0, -2.0], device=D)
        return dict(sh=torch.randn(333, 3, 16, device=D, generator=_gen(8)), xyz=torch.randn(333, 3, device=D, generator=_gen(9))), \
            lambda sh, xyz: (sh_colors(3, sh, xyz, cam),)
    yield "sh", sh

    def bind2(scale=True, per_gaussian=False):
        v, f = _mesh()
        bc, rad = barycentric_table(6, D)
        if per_gaussian:
            bc = torch.rand(f.shape[0], 6, 3, device=D, generator=_gen(10))
        t = dict(verts=v)
        if scale:
            t["scale_factor"] = torch.full((1,), 0.5, device=D)
        return t, lambda verts, scale_factor=None: bind_faces(verts, f, bc, scale_factor, rad, 1.3)
    yield "bind2", bind2
    yield "bind2-no-scale", lambda: bind2(scale=False)
    yield "bind2-per-gaussian", lambda: bind2(per_gaussian=True)

    def bind3():
        v, f = _mesh()
        bc, _ = barycentric_table(3, D)
        n = f.shape[0] * 3
        return dict(verts=v, s2=0.1 * torch.randn(n, 2, device=D, generator=_gen(11)), r2=torch.randn(n, 2, device=D, generator=_gen(12))), \
            lambda verts, s2, r2: bind_faces_scale_rot(verts, f, bc, s2, r2, 1e-5)
    yield "bind3", bind3

    def tex():
        torch.manual_seed(3)
        m = MLPTexture3D(torch.tensor([[-1.0] * 3, [1.0] * 3]), channels=12, device=D)
        with torch.no_grad():
            m.encoder.params.copy_(torch.randn(m.encoder.params.shape, device=D, generator=_gen(13)))
        p = dict(m.named_parameters())
        x = 2 * torch.rand(501, 3, device=D, generator=_gen(14)) - 1
        return dict(xyz=x, **{"p%d" % i: q for i, q in enumerate(p.values())}), lambda xyz, **_: (m.sample_noact(xyz),)
    yield "texture", tex

    def fc(weights):
        c = FlexiCubes(device=D)
        res = (9, 8, 10)
        grid, cubes = c.construct_voxel_grid_v2(res, [-1.0] * 3, [1.0] * 3)
        s = torch.randn(grid.shape[0], device=D, generator=_gen(15)) + 3 * (grid.norm(dim=1) - 0.6)
        t = dict(x=grid + 0.02 * torch.randn(grid.shape, device=D, generator=_gen(16)), s=s)
        if weights == "fused":
            t["w"] = torch.randn(cubes.shape[0], 21, device=D, generator=_gen(17))
            return t, lambda x, s, w: c(x, s, cubes, res, w[:, :12], w[:, 12:20], w[:, 20], training=True)
        if weights == "apart":
            n = cubes.shape[0]
            t.update(b=torch.randn(n, 12, device=D, generator=_gen(18)), a=torch.randn(n, 8, device=D, generator=_gen(19)),
                     g=torch.randn(n, device=D, generator=_gen(20)))
            return t, lambda x, s, b, a, g: c(x, s, cubes, res, b, a, g)
        return t, lambda x, s: c(x, s, cubes, res)
    for w in ("fused", "apart", "none"):
        yield "flexicubes-" + w, lambda w=w: fc(w)


OPS = dict(_ops())


def _run(make, twice=False, hooks=None):
    tensors, fn = make()
    for t in tensors.values():
        t.requires_grad_(True)
    if hooks is None:
        outs = fn(**tensors)
    else:
        with hooks:
            outs = fn(**tensors)
    diff = [o for o in outs if o is not None and o.requires_grad]
    d = [torch.randn(o.shape, device=D, generator=_gen(99)) for o in diff]
    grads = torch.autograd.grad(diff, list(tensors.values()), d, allow_unused=True, retain_graph=twice)
    if twice:
        grads = torch.autograd.grad(diff, list(tensors.values()), d, allow_unused=True)
    return [None if o is None else o.detach() for o in outs], [o.requires_grad for o in outs if o is not None], grads


def _same(a, b):
    for x, y in zip(a[0], b[0]):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.dtype == y.dtype and torch.equal(x, y)
    assert a[1] == b[1]
    for x, y in zip(a[2], b[2]):
        assert (x is None) == (y is None)
        if x is not None:  # sums by float atomics: run-to-run rounding
            assert x.shape == y.shape and float((x - y).norm()) <= 1e-5 * float(y.norm()) + 1e-12


@pytest.mark.parametrize("op", list(OPS))
def test_native_and_general_forms_agree(op, monkeypatch):
    took = []
    real = _lib.native_call
    monkeypatch.setattr(_lib, "native_call", lambda name, *a: took.append(real(name, *a)) or took[-1])
    native = _run(OPS[op])
    assert took[-1] is not None  # the native node took the call
    again = _run(OPS[op], twice=True)
    offloaded = _run(OPS[op], hooks=torch.autograd.graph.save_on_cpu())
    monkeypatch.setattr(_lib, "native_call", lambda name, *a: None)
    general = _run(OPS[op])
    _same(native, general)
    _same(again, general)
    _same(offloaded, general)


@pytest.mark.parametrize("op", list(OPS))
def test_other_dtypes_and_strides_take_the_general_form(op, monkeypatch):
    def strided():
        t, fn = OPS[op]()
        name = next(k for k in t if k not in ("means2D",) and not k.startswith("p"))
        x = t[name]
        if x.dim() > 1:
            t[name] = x.detach().transpose(0, 1).contiguous().transpose(0, 1)
        else:
            t[name] = x.detach().double()
        return t, fn
    took = []
    real = _lib.native_call
    monkeypatch.setattr(_lib, "native_call", lambda name, *a: took.append(real(name, *a)) or took[-1])
    a = _run(strided)
    assert took[-1] is None
    b = _run(OPS[op])
    for x, y in zip(a[0], b[0]):
        if x is not None:
            assert torch.equal(x, y)
    for x, y in zip(a[2], b[2]):
        if x is not None:
            assert float((x - y).norm()) <= 1e-5 * float(y.norm()) + 1e-12


def test_errors_keep_their_type():
    g, _ = _raster("sh")
    sc = small_scene(P=4, width=16, height=16)
    v = sc.views[0]
    rs = dmgs_gb300.GaussianRasterizationSettings(
        image_height=16, image_width=16, tanfovx=v.tanfovx, tanfovy=v.tanfovy, bg=torch.zeros(3, device=D), scale_modifier=1.0,
        viewmatrix=torch.tensor(v.viewmatrix, device=D), projmatrix=torch.tensor(v.projmatrix, device=D), sh_degree=7,
        campos=torch.tensor(v.campos, device=D), prefiltered=False, debug=False)
    with pytest.raises(DmgsError) as e:
        dmgs_gb300.GaussianRasterizer(rs)(**g)
    assert e.value.code == -1 and "sh_degree" in str(e.value)
    with pytest.raises(RuntimeError, match="num_points, 3"):
        dmgs_gb300.GaussianRasterizer(rs)(**{**g, "means3D": g["means3D"][:, :2]})
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        dmgs_gb300.GaussianRasterizer(rs)(**{k: t.cpu() for k, t in g.items()})
    assert np.isfinite(g["means3D"].cpu().numpy()).all()
