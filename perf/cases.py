"""The work this framework is timed on, through its public entry points.

Every case is a dict of plain values.  ``kind`` names the entry point:

  fit      BatchRenderer.render_l1(..., grads_in_forward=True) on clip_space_packed
           positions, backward to vertices and attributes (an image-fitting step);
  render   BatchRenderer(pos, attr) without gradients (rendering many items);
  chain    rasterize -> interpolate -> antialias -> l1_loss through the drop-in
           ``nvdr`` calls with a batch of views, backward to clip positions and
           attributes (an unmodified diffrp / nvdiffrast program);
  raster   DepthPeeler layers with rast_db, forward and backward;
  interp   interpolate with screen-space derivatives, forward and backward;
  aa       antialias, forward and backward;
  texture  texture sampling, forward and backward;
  session  the README example through SurfaceDeferredRenderSession.

``exact`` restates the same mathematics in plain torch float64.  Which triangle a
pixel shows is a decision on whole numbers (fixed-point edge functions, a 64-bit
depth key), restated below in whole numbers too; everything that is a value is
float64.
"""
import functools
import math

import numpy as np
import torch

from diffrp_gb300 import nvdr as dr
from diffrp_gb300 import synthetic
from diffrp_gb300.batch import BatchRenderer
from diffrp_gb300.losses import l1_loss
from diffrp_gb300.transform import clip_space_packed

DEV = "cuda"


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest fitting step: one low-resolution view of a small mesh, captured as one CUDA
        # graph as fitting loops are; launches and latency are all there is
        dict(name="fit_tiny_graph", kind="fit", mesh="ico", detail=3, views=1, height=256, width=256, channels=4,
             tile=4, tpt=0, graph=True, recompute=False),
        # the benchmark's headline: 20480 triangles, one 1024x1024 view, 8 channels, one CUDA graph
        dict(name="fit_single_graph", kind="fit", mesh="ico", detail=5, views=1, height=1024, width=1024, channels=8,
             tile=5, tpt=0, graph=True, recompute=False),
        # multi-view fitting: 64 views of one mesh in one launch sequence
        dict(name="fit_views", kind="fit", mesh="ico", detail=3, views=64, height=512, width=512, channels=8,
             tile=5, tpt=0, graph=False, recompute=False),
        # a mesh of millions of triangles at high resolution, rendered in chunks (the raster shape the
        # autotuner picks for it)
        dict(name="fit_heightfield", kind="fit", mesh="grid", detail=1024, views=4, height=2048, width=2048,
             channels=12, tile=5, tpt=1, graph=False, recompute=True),
        # rendering only: meshes of 1e3 to 3e5 triangles, ragged resolutions, 4 to 16 channels
        dict(name="render_uneven", kind="render", meshes=10, layout=1, res_min=200, res_max=1100, tile=4, tpt=0),
        # an unmodified program on the drop-in calls: six views at an odd resolution, topology
        # rebuilt by every antialias call as diffrp's own call does
        dict(name="chain_views", kind="chain", mesh="ico", detail=5, views=6, height=800, width=1000, channels=8),
        # depth peeling with screen-space derivatives at full HD, two layers, forward and backward
        dict(name="raster_peel", kind="raster", mesh="ico", detail=6, height=1080, width=1920, layers=2),
        # varyings of a textured material (uv and a normal), with uv derivatives
        dict(name="interp_uv_normal", kind="interp", mesh="ico", detail=5, views=4, height=1024, width=1024,
             channels=5, diff=2),
        # silhouette gradients of shaded RGB images, eight views
        dict(name="aa_rgb", kind="aa", mesh="ico", detail=4, views=8, height=512, width=512, channels=3),
        # the benchmark's texture workload: RGBA, trilinear, a ground plane tiled many times
        dict(name="texture_rgba", kind="texture", tex_n=1, tex_h=1024, tex_w=1024, channels=4, views=1, height=1024,
             width=1024, filter="linear-mipmap-linear", boundary="wrap", tiles=16.0),
        # an RGB albedo map of odd size seen close up, two views
        dict(name="texture_rgb_odd", kind="texture", tex_n=1, tex_h=750, tex_w=1000, channels=3, views=2, height=500,
             width=700, filter="linear-mipmap-linear", boundary="mirror", tiles=2.0),
        # the README example (forward): scene and session built anew, flat normals, antialiased
        dict(name="session_normals", kind="session", detail=3, height=512, width=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "render", "chain", "raster", "interp", "aa", "texture", "texture", "session"])
    if kind == "fit":
        h, w = _log(rng, 200, 1600), _log(rng, 200, 1600)
        views = max(1, min(_log(rng, 1, 64), 16000000 // (h * w)))
        big = rng.random() < 0.3
        return dict(kind=kind, mesh="grid" if big else "ico", detail=_log(rng, 24, 700) if big else rng.randint(3, 6),
                    views=views, height=h, width=w, channels=rng.randint(3, 16), tile=rng.choice([4, 5]), tpt=rng.choice([0, 1]) if big else 0,
                    graph=rng.random() < 0.5, recompute=rng.random() < 0.2)
    if kind == "render":
        top = _log(rng, 300, 1100)
        return dict(kind=kind, meshes=rng.randint(2, 12), layout=rng.randint(2, 10 ** 6), res_min=max(64, top // 5),
                    res_max=top, tile=rng.choice([4, 5]), tpt=0)
    if kind == "session":
        return dict(kind=kind, detail=rng.randint(2, 5), height=_log(rng, 200, 1100), width=_log(rng, 200, 1100))
    if kind == "texture":
        h, w = _log(rng, 150, 1400), _log(rng, 150, 1400)
        views = rng.randint(1, 4)
        return dict(kind=kind, tex_n=rng.choice([1, views]), tex_h=_log(rng, 64, 1500), tex_w=_log(rng, 64, 1500),
                    channels=rng.randint(1, 6), views=views, height=h, width=w,
                    filter=rng.choice(["linear", "linear-mipmap-linear", "linear-mipmap-linear"]),
                    boundary=rng.choice(["wrap", "clamp", "zero", "mirror"]), tiles=math.exp(rng.uniform(0.0, 2.8)))
    h, w = _log(rng, 200, 1500), _log(rng, 200, 1500)
    if kind == "raster":
        return dict(kind=kind, mesh="ico", detail=rng.randint(3, 6), height=h, width=w, layers=rng.randint(1, 3))
    views = max(1, min(_log(rng, 1, 12), 6000000 // (h * w)))
    base = dict(kind=kind, mesh="ico", detail=rng.randint(3, 6), views=views, height=h, width=w,
                channels=rng.randint(1, 12))
    if kind == "interp":
        base["diff"] = rng.randint(0, min(4, base["channels"]))
    return base


# ---------------------------------------------------------------------------
# Inputs, from the seed alone
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _base_mesh(kind, detail):
    if kind == "ico":
        v, f = synthetic.icosphere(detail, 0.8)
    else:
        v, f = synthetic.grid_mesh(detail)
    return torch.from_numpy(v).to(DEV), torch.from_numpy(f).to(DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _mesh(kind, detail, g):
    """Displaced icosphere (radial normal noise) or heightfield (a sum of
    waves with random phases), (V, 3) float32 and (F, 3) int32."""
    v, f = _base_mesh(kind, detail)
    if kind == "ico":
        sigma = min(0.02, 0.44 / 2 ** detail)
        return v + v / 0.8 * (sigma * torch.randn((len(v), 1), generator=g, device=DEV)), f
    ph = 2 * math.pi * torch.rand((6, 3), generator=g, device=DEV)
    z = torch.zeros(len(v), device=DEV)
    for k in range(6):
        fr = 2.0 ** k
        z = z + 0.12 * 0.5 ** k * (torch.sin(2.1 * fr * v[:, 0] + ph[k, 0]) * torch.sin(1.7 * fr * v[:, 1] + ph[k, 1])
                                   + 0.5 * torch.sin(1.3 * fr * (v[:, 0] + v[:, 1]) + ph[k, 2]))
    v = v.clone()
    v[:, 2] = z
    return v, f


def _mvps(kind, views, h, w, seed):
    """(views, 4, 4) float32: eyes on a sphere around an icosphere, or an
    oblique ring around a heightfield."""
    rng = np.random.default_rng(seed)
    out = []
    if kind == "ico":
        P = synthetic.perspective(30.0, h, w, 0.1, 100.0).astype(np.float64)
        for e in synthetic.sphere_eyes(views, 3.2, seed=int(rng.integers(1 << 30))):
            out.append(P @ synthetic.view_matrix(synthetic.lookat_pose(e)).astype(np.float64))
    else:
        P = synthetic.perspective(40.0, h, w, 0.1, 20.0).astype(np.float64)
        az0 = rng.uniform(0, 2 * np.pi)
        for k in range(views):
            az = az0 + 2 * np.pi * k / max(views, 1)
            el = np.radians(35.0 + 10.0 * np.sin(3 * az))
            eye = 2.6 * np.array([np.cos(az) * np.cos(el), np.sin(az) * np.cos(el), np.sin(el)])
            out.append(P @ synthetic.view_matrix(synthetic.lookat_pose(eye, up=(0.0, 0.0, 1.0))).astype(np.float64))
    return torch.from_numpy(np.stack(out).astype(np.float32)).to(DEV)


def _uneven_layout(case):
    """(mesh kind, detail, channels, [(height, width)]) per mesh."""
    rng = np.random.default_rng(case["layout"])
    out = []
    for _ in range(case["meshes"]):
        F = math.exp(rng.uniform(math.log(1e3), math.log(3e5)))
        ico = rng.uniform() < 0.5
        detail = int(np.clip(round(math.log(F / 20.0) / math.log(4.0)), 3, 6)) if ico else int(round(math.sqrt(F / 2))) + 1
        c = int(rng.integers(4, 17))
        res = [(int(math.exp(rng.uniform(math.log(case["res_min"]), math.log(case["res_max"])))),
                int(math.exp(rng.uniform(math.log(case["res_min"]), math.log(case["res_max"])))))
               for _ in range(int(rng.integers(1, 4)))]
        out.append(("ico" if ico else "grid", detail, c, res))
    return out


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV)


def _clip32(verts, mvps):
    """Clip positions (B, V, 4) float32 of (V, 3) vertices: the chain of fused
    multiply-adds x, y, z onto the translation, each rounded to float32."""
    m = mvps.double()[:, None]
    v = verts.double()[None]
    acc = (v[..., 0:1] * m[..., :, 0] + m[..., :, 3]).float().double()
    acc = (v[..., 1:2] * m[..., :, 1] + acc).float().double()
    return (v[..., 2:3] * m[..., :, 2] + acc).float()


def _inputs(case, seed):
    g = _gen(seed)
    k = case["kind"]
    if k == "fit":
        v, f = _mesh(case["mesh"], case["detail"], g)
        B, H, W, C = case["views"], case["height"], case["width"], case["channels"]
        return dict(verts=v, tri=f, mvps=_mvps(case["mesh"], B, H, W, seed), attr=_rand(g, len(v), C),
                    target=_rand(g, B * H * W * C))
    if k == "render":
        meshes, items = [], []
        for m, (mk, detail, c, res) in enumerate(_uneven_layout(case)):
            v, f = _mesh(mk, detail, g)
            meshes.append((v, f, _rand(g, len(v), c)))
            for j, (h, w) in enumerate(res):
                items.append((m, (h, w), _clip32(v, _mvps(mk, 1, h, w, seed + 7919 * m + j))[0]))
        return dict(meshes=meshes, items=items)
    if k == "texture":
        H, W, N = case["height"], case["width"], case["views"]
        Y, X = torch.meshgrid((2 * torch.arange(H, device=DEV, dtype=torch.float64) + 1) / H - 1,
                              (2 * torch.arange(W, device=DEV, dtype=torch.float64) + 1) / W - 1, indexing="ij")
        uvs, das = [], []
        for n in range(N):  # a plane receding from depth 1 to 16, turned by a seeded angle
            r = torch.rand(3, generator=g, device=DEV).double().tolist()
            a = 0.6 * (r[0] - 0.5)
            q = 17 / 32 - Y * 15 / 32
            pu = case["tiles"] * (math.cos(a) * X - math.sin(a) * Y + r[1]) / 4
            pv = case["tiles"] * (math.sin(a) * X + math.cos(a) * Y + r[2])
            dux, duy = case["tiles"] * math.cos(a) / 4, -case["tiles"] * math.sin(a) / 4
            dvx, dvy = case["tiles"] * math.sin(a), case["tiles"] * math.cos(a)
            dqy = -15 / 32
            uvs.append(torch.stack([pu / q / 4, pv / q / 4], -1))
            das.append(torch.stack([dux / q / 4 * 2 / W, (duy - pu / q * dqy) / q / 4 * 2 / H, dvx / q / 4 * 2 / W,
                                    (dvy - pv / q * dqy) / q / 4 * 2 / H], -1))
        mip = case["filter"].startswith("linear-mipmap")
        return dict(tex=_rand(g, case["tex_n"], case["tex_h"], case["tex_w"], case["channels"]),
                    uv=torch.stack(uvs).float().contiguous(),
                    da=torch.stack(das).float().contiguous() if mip else None,
                    gout=_randn(g, N, H, W, case["channels"]))
    if k == "session":
        v, f = _mesh("ico", case["detail"], g)
        return dict(verts=v, tri=f)
    H, W = case["height"], case["width"]
    v, f = _mesh(case["mesh"], case["detail"], g)
    if k == "raster":
        L = case["layers"]
        return dict(pos=_clip32(v, _mvps(case["mesh"], 1, H, W, seed))[0], tri=f,
                    g_rast=[_randn(g, 1, H, W, 4) for _ in range(L)], g_db=[_randn(g, 1, H, W, 4) for _ in range(L)])
    B, C = case["views"], case["channels"]
    pos = _clip32(v, _mvps(case["mesh"], B, H, W, seed)).contiguous()
    if k == "chain":
        return dict(pos=pos, tri=f, attr=_rand(g, len(v), C), target=_rand(g, B, H, W, C))
    with torch.no_grad():
        layers = [_shade(pos[b].double(), f, _visible(pos[b], f, H, W)[0], H, W, k == "interp") for b in range(B)]
    d = dict(pos=pos, tri=f, rast=torch.stack([r for r, _ in layers]).float())
    if k == "interp":
        d.update(attr=_rand(g, len(v), C), db=torch.stack([x for _, x in layers]).float(),
                 g_out=_randn(g, B, H, W, C), g_da=_randn(g, B, H, W, 2 * case["diff"]))
    else:
        d.update(color=_rand(g, B, H, W, C), g_out=_randn(g, B, H, W, C))
    return d


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _leaf(t):
    return t.detach().clone().requires_grad_(True)


def _fit_step(s):
    s["verts"].grad = s["attr"].grad = None
    pos = clip_space_packed([(s["verts"], s["mvps"])])
    loss, images = s["renderer"].render_l1(pos, s["attr"].reshape(-1), s["target"], grads_in_forward=True)
    loss.backward()
    return dict(loss=loss.detach(), images=images.detach(), g_verts=s["verts"].grad, g_attr=s["attr"].grad)


def prepare(case, seed):
    k = case["kind"]
    d = _inputs(case, seed)
    s = dict(case=case)
    if k == "fit":
        s.update(verts=_leaf(d["verts"]), attr=_leaf(d["attr"]), mvps=d["mvps"], target=d["target"])
        s["renderer"] = BatchRenderer([(d["tri"], len(d["verts"]), case["channels"])],
                                      [(0, (case["height"], case["width"]))] * case["views"], tile_log2=case["tile"],
                                      threads_per_tri=case["tpt"], recompute=case["recompute"])
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                for _ in range(3):
                    _fit_step(s)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            s["replay"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["replay"]):
                s["outputs"] = _fit_step(s)
        return s
    if k == "render":
        s["renderer"] = BatchRenderer([(f, len(v), a.shape[1]) for v, f, a in d["meshes"]],
                                      [(m, hw) for m, hw, _ in d["items"]], tile_log2=case["tile"],
                                      threads_per_tri=case["tpt"])
        s["pos"] = s["renderer"].pack_positions([p for _, _, p in d["items"]])
        s["attr"] = s["renderer"].pack_attributes([a for _, _, a in d["meshes"]])
        return s
    if k == "session":
        from diffrp_gb300.rendering.camera import PerspectiveCamera
        s.update(verts=d["verts"], tri=d["tri"],
                 camera=PerspectiveCamera(h=case["height"], w=case["width"], far=100.0))
        return s
    if k == "texture":
        s.update(tex=_leaf(d["tex"]), uv=_leaf(d["uv"]), da=None if d["da"] is None else _leaf(d["da"]),
                 gout=d["gout"])
        return s
    s.update(d)
    if k in ("chain", "raster"):
        s["ctx"] = dr.RasterizeCudaContext()
    for name in {"chain": ("pos", "attr"), "raster": ("pos",), "interp": ("attr", "rast", "db"),
                 "aa": ("pos", "color")}[k]:
        s[name] = _leaf(d[name])
    if k == "aa":
        s["topology"] = dr.antialias_construct_topology_hash(d["tri"])
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "fit":
        if "replay" in s:
            s["replay"].replay()
            return s["outputs"]
        return _fit_step(s)
    if k == "render":
        with torch.no_grad():
            return s["renderer"](s["pos"], s["attr"])
    if k == "chain":
        hw = (case["height"], case["width"])
        rast, _ = dr.rasterize(s["ctx"], s["pos"], s["tri"], hw, grad_db=False)
        color, _ = dr.interpolate(s["attr"], rast, s["tri"])
        img = dr.antialias(color, rast, s["pos"], s["tri"])
        loss = l1_loss(img, s["target"])
        g_pos, g_attr = torch.autograd.grad(loss, (s["pos"], s["attr"]))
        return dict(loss=loss.detach(), images=img.detach(), g_pos=g_pos, g_attr=g_attr)
    if k == "raster":
        outs = []
        with dr.DepthPeeler(s["ctx"], s["pos"], s["tri"], (case["height"], case["width"])) as peeler:
            for _ in range(case["layers"]):
                outs.append(peeler.rasterize_next_layer())
        g_pos, = torch.autograd.grad([r for r, _ in outs] + [db for _, db in outs], (s["pos"],),
                                     s["g_rast"] + s["g_db"])
        return dict(rast=[r.detach() for r, _ in outs], db=[db.detach() for _, db in outs], g_pos=g_pos)
    if k == "interp":
        if case["diff"]:
            out, da = dr.interpolate(s["attr"], s["rast"], s["tri"], rast_db=s["db"],
                                     diff_attrs=list(range(case["diff"])))
            g_attr, g_rast, g_db = torch.autograd.grad((out, da), (s["attr"], s["rast"], s["db"]),
                                                       (s["g_out"], s["g_da"]))
            return dict(out=out.detach(), da=da.detach(), g_attr=g_attr, g_rast=g_rast, g_db=g_db)
        out, _ = dr.interpolate(s["attr"], s["rast"], s["tri"])
        g_attr, g_rast = torch.autograd.grad(out, (s["attr"], s["rast"]), s["g_out"])
        return dict(out=out.detach(), g_attr=g_attr, g_rast=g_rast)
    if k == "aa":
        img = dr.antialias(s["color"], s["rast"], s["pos"], s["tri"], topology_hash=s["topology"])
        g_color, g_pos = torch.autograd.grad(img, (s["color"], s["pos"]), s["g_out"])
        return dict(images=img.detach(), g_color=g_color, g_pos=g_pos)
    if k == "texture":
        leaves = [s["tex"], s["uv"]] + ([s["da"]] if s["da"] is not None else [])
        out = dr.texture(s["tex"], s["uv"], s["da"], filter_mode=case["filter"], boundary_mode=case["boundary"])
        grads = torch.autograd.grad(out, leaves, s["gout"])
        return dict(out=out.detach(), grads=list(grads))
    from diffrp_gb300.materials import DefaultMaterial
    from diffrp_gb300.rendering.surface_deferred import SurfaceDeferredRenderSession
    from diffrp_gb300.scene import MeshObject, Scene
    with torch.no_grad():
        scene = Scene().add_mesh_object(MeshObject(DefaultMaterial(), s["verts"], s["tri"]))
        rp = SurfaceDeferredRenderSession(scene, s["camera"])
        return rp.nvdr_antialias(rp.false_color_camera_space_normal()[..., :3])


# ---------------------------------------------------------------------------
# work: each input read once, each output written once
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _mesh_size(kind, detail):
    if kind == "ico":
        return 10 * 4 ** detail + 2, 20 * 4 ** detail
    return detail * detail, 2 * (detail - 1) ** 2


def work(case):
    k = case["kind"]
    if k == "render":
        b = fl = 0
        for mk, detail, c, res in _uneven_layout(case):
            V, F = _mesh_size(mk, detail)
            px = sum(h * w for h, w in res)
            b += V * 4 * c + F * 12 + len(res) * V * 16 + px * 4 * c
            fl += len(res) * F * 60 + px * (60 + 4 * c)
        return dict(bytes=b, flops=fl)
    px = case["height"] * case["width"] * case.get("views", 1)
    if k == "texture":
        C, T = case["channels"], case["tex_n"] * case["tex_h"] * case["tex_w"] * case["channels"]
        da = 32 if case["filter"].startswith("linear-mipmap") else 0
        taps = 8 if da else 4
        return dict(bytes=8 * T + px * (8 + 8 + da + 8 * C), flops=px * taps * C * 6)
    V, F = _mesh_size(case.get("mesh", "ico"), case["detail"])
    if k == "session":
        return dict(bytes=V * 12 + F * 12 + px * 12, flops=F * 100 + px * 100)
    if k == "raster":
        L = case["layers"]
        return dict(bytes=V * 32 + F * 12 + px * 64 * L, flops=F * 60 + px * 250 * L)
    B, C = case["views"], case["channels"]
    if k == "fit":
        return dict(bytes=V * 24 + V * 8 * C + F * 12 + B * 64 + px * 8 * C, flops=B * F * 60 + px * (160 + 16 * C))
    if k == "chain":
        return dict(bytes=B * V * 32 + V * 8 * C + F * 12 + px * 8 * C, flops=B * F * 60 + px * (160 + 16 * C))
    if k == "interp":
        D = case["diff"]
        return dict(bytes=V * 8 * C + F * 12 + px * (16 + 16 + 8 * C + (32 if D else 0) + 16 * D),
                    flops=px * (14 * C + 20 * D))
    return dict(bytes=B * V * 32 + 2 * F * 12 + px * (16 + 16 * C), flops=B * F * 60 + px * (40 + 6 * C))


# ---------------------------------------------------------------------------
# exact: plain torch in 64 bits
# ---------------------------------------------------------------------------
def _visible(pos, tri, H, W, layers=1):
    """Triangle index per pixel, -1 for none, of the nearest `layers` layers:
    (layers, H, W) int64.  Vertices snapped to 1/256 pixel (float32, nearest
    even), exact edge functions with the top-left rule, the float32 depth
    plane, the smallest (depth, triangle) key.  Every triangle in front of the
    near plane and inside the guard band (as all scenes here are)."""
    t = tri.long()
    p = pos[t]
    X = torch.round((p[..., 0] / p[..., 3] + 1.0) * float(W * 128)).long()
    Y = torch.round((p[..., 1] / p[..., 3] + 1.0) * float(H * 128)).long()
    Z = p[..., 2] / p[..., 3]
    area = (X[:, 1] - X[:, 0]) * (Y[:, 2] - Y[:, 0]) - (Y[:, 1] - Y[:, 0]) * (X[:, 2] - X[:, 0])
    det = area.float()
    dx1, dy1 = (X[:, 1] - X[:, 0]).float(), (Y[:, 1] - Y[:, 0]).float()
    dx2, dy2 = (X[:, 2] - X[:, 0]).float(), (Y[:, 2] - Y[:, 0]).float()
    dz1, dz2 = Z[:, 1] - Z[:, 0], Z[:, 2] - Z[:, 0]
    A = (dz1 * dy2 - dy1 * dz2) / det
    Bc = (dx1 * dz2 - dz1 * dx2) / det
    x0 = (-((128 - X.amin(1)) >> 8)).clamp(min=0)
    x1 = ((X.amax(1) - 128) >> 8).clamp(max=W - 1)
    y0 = (-((128 - Y.amin(1)) >> 8)).clamp(min=0)
    y1 = ((Y.amax(1) - 128) >> 8).clamp(max=H - 1)
    bw = (x1 - x0 + 1).clamp(min=0)
    n = torch.where(area != 0, bw * (y1 - y0 + 1).clamp(min=0), torch.zeros_like(bw))
    flip = area < 0
    vx = torch.stack([X[:, 0], torch.where(flip, X[:, 2], X[:, 1]), torch.where(flip, X[:, 1], X[:, 2])], 1)
    vy = torch.stack([Y[:, 0], torch.where(flip, Y[:, 2], Y[:, 1]), torch.where(flip, Y[:, 1], Y[:, 2])], 1)
    ends = torch.cumsum(n, 0)
    pix_parts, key_parts = [], []
    step = 1 << 18
    for lo in range(0, len(t), step):
        hi = min(len(t), lo + step)
        nn = n[lo:hi]
        owner = torch.repeat_interleave(torch.arange(lo, hi, device=pos.device), nn)
        if not len(owner):
            continue
        r = torch.arange(len(owner), device=pos.device) - (ends[owner] - n[owner] - (ends[lo] - n[lo]))
        px, py = x0[owner] + r % bw[owner], y0[owner] + r // bw[owner]
        sx, sy = px * 256 + 128, py * 256 + 128
        inside = torch.ones_like(px, dtype=torch.bool)
        for a, b in ((1, 2), (2, 0), (0, 1)):
            ex, ey = (vx[:, b] - vx[:, a])[owner], (vy[:, b] - vy[:, a])[owner]
            e = ex * (sy - vy[owner, a]) - ey * (sx - vx[owner, a])
            inside &= (e > 0) | ((e == 0) & ((ey < 0) | ((ey == 0) & (ex < 0))))
        owner, sx, sy, px, py = owner[inside], sx[inside], sy[inside], px[inside], py[inside]
        z = (Z[owner, 0] + A[owner] * (sx - X[owner, 0]).float()) + Bc[owner] * (sy - Y[owner, 0]).float()
        ok = (z >= -1.0) & (z <= 1.0)
        bits = z[ok].view(torch.int32).long() & 0xffffffff
        order = torch.where(bits >= 1 << 31, 0xffffffff - bits, bits + (1 << 31)) - (1 << 31)
        key_parts.append((order << 32) | owner[ok])
        pix_parts.append((py * W + px)[ok])
    top = (1 << 63) - 1
    out, prev = [], None
    pix = torch.cat(pix_parts) if pix_parts else torch.zeros(0, dtype=torch.int64, device=pos.device)
    key = torch.cat(key_parts) if key_parts else torch.zeros(0, dtype=torch.int64, device=pos.device)
    for _ in range(layers):
        if prev is not None:
            later = key > prev[pix]
            pix, key = pix[later], key[later]
        best = torch.full((H * W,), top, dtype=torch.int64, device=pos.device)
        best.scatter_reduce_(0, pix, key, "amin")
        out.append(torch.where(best == top, torch.full_like(best, -1), best & 0xffffffff).view(H, W))
        prev = best
    return torch.stack(out)


def _shade(pos, tri, ids, H, W, want_db=False):
    """rast (H, W, 4) and rast_db (H, W, 4) float64 of the triangles `ids`
    shows: barycentrics in 2D homogeneous coordinates at the pixel centre."""
    py, px = torch.nonzero(ids >= 0, as_tuple=True)
    t = ids[py, px]
    p = pos[tri.long()[t]]
    X, Y = ((2 * px + 1).double() / W - 1)[:, None], ((2 * py + 1).double() / H - 1)[:, None]
    a, c, w = p[..., 0] - X * p[..., 3], p[..., 1] - Y * p[..., 3], p[..., 3]
    n = torch.linalg.cross(a, c)
    s = n.sum(-1)
    u, v = n[:, 0] / s, n[:, 1] / s
    zw = (n * p[..., 2]).sum(-1) / (n * w).sum(-1)
    rast = torch.zeros((H, W, 4), dtype=torch.float64, device=pos.device)
    rast = rast.index_put((py, px), torch.stack([u, v, zw, (t + 1).double()], -1))
    if not want_db:
        return rast, None
    Dx, Dy = torch.linalg.cross(c, w), torch.linalg.cross(w, a)
    Sx, Sy = Dx.sum(-1), Dy.sum(-1)
    d = torch.stack([(Dx[:, 0] - u * Sx) / s * 2 / W, (Dy[:, 0] - u * Sy) / s * 2 / H,
                     (Dx[:, 1] - v * Sx) / s * 2 / W, (Dy[:, 1] - v * Sy) / s * 2 / H], -1)
    db = torch.zeros((H, W, 4), dtype=torch.float64, device=pos.device).index_put((py, px), d)
    return rast, db


def _interp(attr, tri, rast, ids, db=None, diff=0):
    H, W = ids.shape
    py, px = torch.nonzero(ids >= 0, as_tuple=True)
    A = attr[tri.long()[ids[py, px]]]
    r = rast[py, px]
    u, v = r[:, 0:1], r[:, 1:2]
    e0, e1 = A[:, 0] - A[:, 2], A[:, 1] - A[:, 2]
    out = torch.zeros((H, W, attr.shape[1]), dtype=torch.float64, device=attr.device)
    out = out.index_put((py, px), e0 * u + e1 * v + A[:, 2])
    if not diff:
        return out, None
    d = db[py, px]
    e0, e1 = e0[:, :diff], e1[:, :diff]
    val = torch.stack([e0 * d[:, 0:1] + e1 * d[:, 2:3], e0 * d[:, 1:2] + e1 * d[:, 3:4]], -1).flatten(1)
    da = torch.zeros((H, W, 2 * diff), dtype=torch.float64, device=attr.device)
    return out, da.index_put((py, px), val)


def _opposite(tri):
    """Per triangle edge (k joins vertices k + 1, k + 2) the other triangle's
    vertex opposite it, -1 unless exactly two triangles share the edge."""
    t = tri.long()
    V = int(t.max()) + 1
    e = torch.stack([torch.stack([t[:, (k + 1) % 3], t[:, (k + 2) % 3]], -1) for k in range(3)], 1).reshape(-1, 2)
    key = e.amin(1) * V + e.amax(1)
    sk, order = torch.sort(key, stable=True)
    first = torch.ones_like(sk, dtype=torch.bool)
    first[1:] = sk[1:] != sk[:-1]
    group = torch.cumsum(first.long(), 0) - 1
    pair = torch.bincount(group)[group] == 2
    a = torch.nonzero(pair & first).squeeze(1)
    opp = torch.full((len(key),), -1, dtype=torch.int64, device=tri.device)
    flat = t.reshape(-1)
    ea, eb = order[a], order[a + 1]
    ok = (ea // 3 != eb // 3) & (e[ea, 0] != e[ea, 1])
    ea, eb = ea[ok], eb[ok]
    opp[ea] = flat[eb]
    opp[eb] = flat[ea]
    return opp.view(-1, 3)


def _antialias(color, ids, zw, pos, tri, opp):
    """Silhouette blend of color (H, W, C) float64, differentiable w.r.t.
    color and pos; ids, zw: triangle and depth per pixel."""
    H, W, C = color.shape
    t = tri.long()
    s = (pos[:, :2] / pos[:, 3:4] + 1) * torch.tensor([W * 0.5, H * 0.5], dtype=torch.float64, device=pos.device)
    flat = ids.reshape(-1)
    zf = zw.reshape(-1)
    lin = torch.arange(H * W, device=pos.device).view(H, W)
    col = color.reshape(H * W, C)
    tgt_all, val_all = [], []

    def edge(a, b, p):
        return (b[:, 0] - a[:, 0]) * (p[:, 1] - a[:, 1]) - (b[:, 1] - a[:, 1]) * (p[:, 0] - a[:, 0])

    for A, B in ((lin[:, :-1], lin[:, 1:]), (lin[:-1], lin[1:])):
        A, B = A.reshape(-1), B.reshape(-1)
        keep = flat[A] != flat[B]
        A, B = A[keep], B[keep]
        cA, cB = flat[A], flat[B]
        front_a = (cB < 0) | ((cA >= 0) & ((zf[A] < zf[B]) | ((zf[A] == zf[B]) & (cA < cB))))
        Fp, Op = torch.where(front_a, A, B), torch.where(front_a, B, A)
        T = flat[Fp]
        cF = torch.stack([Fp % W, Fp // W], -1).double() + 0.5
        cO = torch.stack([Op % W, Op // W], -1).double() + 0.5
        q = s[t[T]]
        area = edge(q[:, 0], q[:, 1], q[:, 2])
        sgn = torch.sign(area).detach()
        eO = torch.stack([sgn * edge(q[:, (k + 1) % 3], q[:, (k + 2) % 3], cO) for k in range(3)], 1)
        eF = torch.stack([sgn * edge(q[:, (k + 1) % 3], q[:, (k + 2) % 3], cF) for k in range(3)], 1)
        with torch.no_grad():
            tt = torch.where(eO < 0, eF / (eF - eO), torch.full_like(eF, math.inf))
            k = tt.argmin(1)
            ok = (sgn != 0) & (eO < 0).any(1)
            r = torch.arange(len(k), device=pos.device)
            ov = opp[T, k]
            qa, qb, qk = q[r, (k + 1) % 3], q[r, (k + 2) % 3], q[r, k]
            fold = edge(qa, qb, qk) * edge(qa, qb, s[ov.clamp(min=0)]) < 0
            ok &= (ov < 0) | ~fold
        r, k = r[ok], k[ok]
        ef, eo = eF[r, k], eO[r, k]
        tv = (ef / (ef - eo)).clamp(0.0, 1.0)
        far = tv.detach() > 0.5
        Fp, Op = Fp[ok], Op[ok]
        tgt, src = torch.where(far, Op, Fp), torch.where(far, Fp, Op)
        tgt_all.append(tgt)
        val_all.append((tv - 0.5).abs()[:, None] * (col[src] - col[tgt]))
    return col.index_put((torch.cat(tgt_all),), torch.cat(val_all), accumulate=True).view(H, W, C)


def _view64(pos64, pos32, tri, attr64, opp, H, W):
    ids = _visible(pos32, tri, H, W)[0]
    rast, _ = _shade(pos64, tri, ids, H, W)
    color, _ = _interp(attr64, tri, rast, ids)
    return _antialias(color, ids, rast[..., 2].detach().float(), pos64, tri, opp)


def _clip64(verts64, mvp):
    m = mvp.double()
    return verts64 @ m[:, :3].T + m[:, 3]


def _texture64(tex, uv, da, mip, boundary):
    """Bilinear / trilinear samples (N, h, w, C) of tex (Nt, H, W, C) float64."""
    Nt, H, W, C = tex.shape
    N, h, w = uv.shape[:3]
    levels = [tex]
    while mip and max(levels[-1].shape[1:3]) > 1:
        q = levels[-1]
        ph, pw = q.shape[1:3]
        y = torch.arange(max(ph >> 1, 1), device=tex.device)
        x = torch.arange(max(pw >> 1, 1), device=tex.device)
        ya, yb = (2 * y).clamp(max=ph - 1), (2 * y + 1).clamp(max=ph - 1)
        xa, xb = (2 * x).clamp(max=pw - 1), (2 * x + 1).clamp(max=pw - 1)
        levels.append((q[:, ya][:, :, xa] + q[:, ya][:, :, xb] + q[:, yb][:, :, xa] + q[:, yb][:, :, xb]) * 0.25)
    lh = torch.tensor([q.shape[1] for q in levels], device=tex.device)
    lw = torch.tensor([q.shape[2] for q in levels], device=tex.device)
    ofs = torch.tensor(np.cumsum([0] + [q.shape[0] * q.shape[1] * q.shape[2] for q in levels[:-1]]), device=tex.device)
    flat = torch.cat([q.reshape(-1, C) for q in levels] + [torch.zeros((1, C), dtype=tex.dtype, device=tex.device)])
    none = len(flat) - 1
    n = torch.arange(N, device=tex.device)[:, None, None] if Nt > 1 else torch.zeros((), dtype=torch.int64,
                                                                                       device=tex.device)

    def index(i, size):
        if boundary == "wrap":
            return i % size, None
        if boundary == "clamp":
            return torch.minimum(i.clamp(min=0), size - 1), None
        if boundary == "mirror":
            m = i % (2 * size)
            return torch.where(m < size, m, 2 * size - 1 - m), None
        return torch.minimum(i.clamp(min=0), size - 1), (i >= 0) & (i < size)

    def bilinear(l):
        H_, W_ = lh[l], lw[l]
        x, y = uv[..., 0] * W_ - 0.5, uv[..., 1] * H_ - 0.5
        x0, y0 = torch.floor(x.detach()), torch.floor(y.detach())
        fx, fy = (x - x0)[..., None], (y - y0)[..., None]
        taps = []
        for dy in (0, 1):
            for dx in (0, 1):
                xi, okx = index(x0.long() + dx, W_)
                yi, oky = index(y0.long() + dy, H_)
                at = ofs[l] + n * (H_ * W_) + yi * W_ + xi
                if okx is not None:
                    at = torch.where(okx & oky, at, torch.full_like(at, none))
                taps.append(flat[at])
        return (taps[0] * (1 - fx) + taps[1] * fx) * (1 - fy) + (taps[2] * (1 - fx) + taps[3] * fx) * fy

    zero = torch.zeros((N, h, w), dtype=torch.int64, device=tex.device)
    if not mip:
        return bilinear(zero)
    ax, bx, ay, by = da[..., 0] * W, da[..., 1] * W, da[..., 2] * H, da[..., 3] * H
    r2 = torch.maximum(ax * ax + ay * ay, bx * bx + by * by)
    lam = (0.5 * torch.log2(r2)).clamp(0.0, len(levels) - 1.0)
    l0 = torch.floor(lam.detach()).long()
    l1 = (l0 + 1).clamp(max=len(levels) - 1)
    f = torch.where(l1 > l0, lam - l0, torch.zeros_like(lam))[..., None]
    return bilinear(l0) * (1 - f) + bilinear(l1) * f


def exact(case, seed):
    k = case["kind"]
    d = _inputs(case, seed)
    if k == "fit":
        H, W, C = case["height"], case["width"], case["channels"]
        verts, attr = _leaf(d["verts"].double()), _leaf(d["attr"].double())
        opp = _opposite(d["tri"])
        pos32 = _clip32(d["verts"], d["mvps"])
        n = d["target"].numel()
        target = d["target"].view(-1, H, W, C)
        loss, images = 0.0, []
        for b in range(case["views"]):
            img = _view64(_clip64(verts, d["mvps"][b]), pos32[b], d["tri"], attr, opp, H, W)
            part = (img - target[b].double()).abs().sum() / n
            part.backward()
            loss = loss + part.detach()
            images.append(img.detach().reshape(-1))
        return dict(loss=loss, images=torch.cat(images), g_verts=verts.grad, g_attr=attr.grad)
    if k == "render":
        out = []
        with torch.no_grad():
            opps = [_opposite(f) for _, f, _ in d["meshes"]]
            for m, (h, w), pos in d["items"]:
                _, f, a = d["meshes"][m]
                out.append(_view64(pos.double(), pos, f, a.double(), opps[m], h, w).reshape(-1))
        return torch.cat(out)
    if k == "texture":
        leaves = [_leaf(d[x].double()) for x in ("tex", "uv", "da") if d[x] is not None]
        out = _texture64(leaves[0], leaves[1], leaves[2] if d["da"] is not None else None, d["da"] is not None,
                         case["boundary"])
        return dict(out=out.detach(), grads=list(torch.autograd.grad(out, leaves, d["gout"].double())))
    H, W = case["height"], case["width"]
    if k == "session":
        with torch.no_grad():
            v = d["verts"][d["tri"].long()]
            soup = v.reshape(-1, 3)
            tri = torch.arange(len(soup), device=DEV, dtype=torch.int32).view(-1, 3)
            pose = np.eye(4)
            pose[2, 3] = 3.2
            V = np.linalg.inv(pose).astype(np.float32)
            VP = torch.from_numpy(synthetic.perspective(30, H, W, 0.1, 100.0)).to(DEV) @ torch.from_numpy(V).to(DEV)
            pos32 = _clip32(soup, VP[None])[0]
            pos = _clip64(soup.double(), VP)
            ids = _visible(pos32, tri, H, W)[0]
            rast, _ = _shade(pos, tri, ids, H, W)
            n = torch.linalg.cross(v[:, 1].double() - v[:, 0].double(), v[:, 2].double() - v[:, 0].double())
            n = n / n.norm(dim=-1, keepdim=True)
            img = torch.where((ids >= 0)[..., None], n[ids.clamp(min=0)], torch.zeros_like(rast[..., :3])) * 0.5 + 0.5
            opp = torch.full((len(tri), 3), -1, dtype=torch.int64, device=DEV)
            return torch.flipud(_antialias(img, ids, rast[..., 2].float(), pos, tri, opp))
    tri = d["tri"]
    if k == "raster":
        pos = _leaf(d["pos"].double())
        ids = _visible(d["pos"], tri, H, W, case["layers"])
        outs = [_shade(pos, tri, i, H, W, True) for i in ids]
        g, = torch.autograd.grad([r for r, _ in outs] + [x for _, x in outs], (pos,),
                                 [x[0].double() for x in d["g_rast"] + d["g_db"]])
        return dict(rast=[r.detach()[None] for r, _ in outs], db=[x.detach()[None] for _, x in outs], g_pos=g)
    B = case["views"]
    if k == "chain":
        pos, attr = _leaf(d["pos"].double()), _leaf(d["attr"].double())
        opp = _opposite(tri)
        n = d["target"].numel()
        loss, images = 0.0, []
        for b in range(B):
            img = _view64(pos[b], d["pos"][b], tri, attr, opp, H, W)
            part = (img - d["target"][b].double()).abs().sum() / n
            part.backward()
            loss = loss + part.detach()
            images.append(img.detach())
        return dict(loss=loss, images=torch.stack(images), g_pos=pos.grad, g_attr=attr.grad)
    ids = d["rast"][..., 3].long() - 1
    if k == "interp":
        D = case["diff"]
        attr, rast, db = (_leaf(d[x].double()) for x in ("attr", "rast", "db"))
        got = [_interp(attr, tri, rast[b], ids[b], db[b], D) for b in range(B)]
        out = torch.stack([o for o, _ in got])
        if not D:
            g = torch.autograd.grad(out, (attr, rast), d["g_out"].double())
            return dict(out=out.detach(), g_attr=g[0], g_rast=g[1])
        da = torch.stack([x for _, x in got])
        g = torch.autograd.grad((out, da), (attr, rast, db), (d["g_out"].double(), d["g_da"].double()))
        return dict(out=out.detach(), da=da.detach(), g_attr=g[0], g_rast=g[1], g_db=g[2])
    pos, color = _leaf(d["pos"].double()), _leaf(d["color"].double())
    opp = _opposite(tri)
    img = torch.stack([_antialias(color[b], ids[b], d["rast"][b, ..., 2], pos[b], tri, opp) for b in range(B)])
    g = torch.autograd.grad(img, (color, pos), d["g_out"].double())
    return dict(images=img.detach(), g_color=g[0], g_pos=g[1])
