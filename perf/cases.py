"""What a user of gstex_cuda_gb300 has it do, as cases that can be timed.

Each case is one call pattern of the package at one size: a training or a
rendering pass of one view through the per-view API (projection, SH, AABBs,
tile counts, ``texture_gaussians``, gradients), a step or a render of many
views through ``BatchRenderer``, texture sampling and editing, and the
trainer's per-step parameter work (activation, SH colours).  Sizes and
distributions are those of ``gstex_cuda_gb300.synthetic``, the tests and the
benchmark; odd ones lie between them.

Scenes: "near" has Gaussians with means in [-1,1]^2 x [2,4] and scales
log-U[0.05,0.5] before a camera at the origin; "cube" has means in [-3,3]^3
and scales log-U[0.005,0.05] seen from distance 8; "clusters" has the same
scales with means in 64 blobs of sigma 0.3.
"""
import math
import random

import torch

from gstex_cuda_gb300 import batch as B
from gstex_cuda_gb300.get_aabb_2d import get_aabb_2d, get_num_tiles_hit_2d, project_points
from gstex_cuda_gb300.preprocess import preprocess
from gstex_cuda_gb300.sh import spherical_harmonics
from gstex_cuda_gb300.texture import texture_gaussians
from gstex_cuda_gb300.texture_edit import texture_edit
from gstex_cuda_gb300.texture_sample import texture_sample

DEV = "cuda:0"
SETTINGS = 1 << 8
LOSS = dict(img=1.0, texture=1.0, reg=100.0, normal=0.05)


def listed():
    return [
        # a unit test or a demo's first picture: 10 splats on 32x32; launches and host calls are all of it
        dict(name="view_tiny", kind="view", scene="near", width=32, height=32, points=10, texels=160, sh_degree=0,
             grad=True),
        # a small training view of odd size, as a crop or a thumbnail
        dict(name="view_ragged", kind="view", scene="near", width=253, height=187, points=2001, texels=60000,
             sh_degree=2, grad=True),
        # the usual training view of an object data set: 800x800, 100k Gaussians without texture detail (1x1 charts)
        dict(name="view_800", kind="view", scene="cube", width=800, height=800, points=100000, texels=0, sh_degree=3,
             grad=True),
        # a full-HD training view with large overlapping splats (over a hundred million tile intersections)
        dict(name="view_1080p", kind="view", scene="near", width=1920, height=1080, points=200000, texels=8000000,
             sh_degree=0, grad=True),
        # showing a trained scene: one 1280x720 picture, no gradients, texels stored as bfloat16
        dict(name="render_720p", kind="view", scene="cube", width=1280, height=720, points=500000, texels=16000000,
             sh_degree=3, grad=False, bf16=True),
        # a trainer's small batch from raw parameters: four views of mixed, odd sizes, float32 texels, stock settings
        dict(name="raw_step_4", kind="batch", scene="cube", sizes="512x512,333x251,640x360,401x603", points=60000,
             texels=1500000, sh_degree=3, bf16=False, raw=True, grad=True, block_width=16, ctas=0),
        # the benchmark's step: 32 views, 500k Gaussians, 16M bf16 texels, with the launch settings its tuner picks
        dict(name="step_32", kind="batch", scene="cube", sizes="512x512*8,800x800*8,1280x720*8,1920x1080*8",
             points=500000, texels=16000000, sh_degree=3, bf16=True, raw=False, grad=True, block_width=8, ctas=10),
        # the benchmark's dense scene: 8 full-HD views of 1M clustered Gaussians
        dict(name="step_clusters", kind="batch", scene="clusters", sizes="1920x1080*8", points=1000000,
             texels=32000000, sh_degree=3, bf16=True, raw=False, grad=True, block_width=8, ctas=10),
        # evaluation on held-out cameras: forward only, stock settings, float32 texels
        dict(name="render_batch_8", kind="batch", scene="cube", sizes="800x800*5,797x533*3", points=200000,
             texels=6000000, sh_degree=3, bf16=False, raw=False, grad=False, block_width=16, ctas=0),
        # lookups in the charts outside the renderer, with their gradients
        dict(name="sample_1m", kind="sample", queries=1000003, charts=50000, side=9, channels=3),
        # painting an edited picture back into the charts
        dict(name="edit_800", kind="edit", scene="cube", width=800, height=800, points=100000, side=4),
        # a training step's per-Gaussian work through the autograd API: activation and SH colours, with gradients
        dict(name="params_500k", kind="params", points=500000, sh_degree=3),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view", "view", "view", "view", "batch", "batch", "batch", "sample", "edit", "params"])
    if kind == "sample":
        return dict(kind=kind, queries=_logu(rng, 1000, 4000000), charts=_logu(rng, 100, 100000),
                    side=rng.randint(1, 16), channels=rng.choice([1, 3, 3, 4]))
    if kind == "params":
        return dict(kind=kind, points=_logu(rng, 1000, 1000000), sh_degree=rng.randint(0, 3))
    scene = rng.choice(["near", "cube", "clusters"])
    points = _logu(rng, 10, 100000) if scene == "near" else _logu(rng, 1000, 500000)
    if kind == "edit":
        return dict(kind=kind, scene=scene, width=_logu(rng, 32, 1280), height=_logu(rng, 32, 1080), points=points,
                    side=rng.randint(1, 8))
    texels = 0 if rng.random() < 0.2 else points * rng.randint(4, 60)
    if kind == "view":
        grad = rng.random() < 0.7
        return dict(kind=kind, scene=scene, width=_logu(rng, 32, 1920), height=_logu(rng, 32, 1080), points=points,
                    texels=texels, sh_degree=rng.randint(0, 3), grad=grad, bf16=not grad and rng.random() < 0.5)
    if scene == "near":
        scene = "cube"
    views = rng.randint(1, 8)
    sizes = ",".join("%dx%d" % (_logu(rng, 64, 1600), _logu(rng, 64, 1080)) for _ in range(views))
    bf16 = rng.random() < 0.6
    bw = rng.choice([8, 16])
    return dict(kind=kind, scene=scene, sizes=sizes, points=max(points, 1000), texels=texels or points,
                sh_degree=rng.randint(0, 3), bf16=bf16, raw=rng.random() < 0.4, grad=rng.random() < 0.7,
                block_width=bw, ctas=10 if bf16 and bw == 8 else 0)


def _sizes(case):
    if case["kind"] != "batch":
        return [(case["width"], case["height"])]
    out = []
    for part in case["sizes"].split(","):
        wh, _, n = part.partition("*")
        w, h = wh.split("x")
        out += [(int(w), int(h))] * int(n or 1)
    return out


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _camera(scene, w, h, r):
    """(viewmat, fx, fy, cx, cy): at the origin for "near", else at distance 8 looking at the centre."""
    if scene == "near":
        f = float(w) if w <= 64 else w / 2.0
        return torch.eye(4, dtype=torch.float64), f, f, w / 2.0, h / 2.0
    c = torch.tensor([r.gauss(0, 1) for _ in range(3)], dtype=torch.float64)
    c = 8.0 * c / c.norm()
    fwd = -c / c.norm()
    up = torch.tensor([0.0, -1.0, 0.0], dtype=torch.float64)
    if abs(float(fwd @ up)) > 0.99:
        up = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64)
    right = torch.linalg.cross(fwd, up)
    right = right / right.norm()
    c2w = torch.eye(4, dtype=torch.float64)
    c2w[:3, :3] = torch.stack([right, torch.linalg.cross(fwd, right), fwd], dim=1)
    c2w[:3, 3] = c
    return torch.linalg.inv(c2w), w / 2.0, w / 2.0, w / 2.0, h / 2.0


def _axes(q):
    w, x, y, z = q.unbind(-1)
    return (torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)], -1),
            torch.stack([2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)], -1),
            torch.stack([2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], -1))


def _scene(case, seed):
    """The scene's tensors, on the GPU.  Charts take texels by projected size
    (2 to 16 a side) from a pool whose size does not depend on the seed."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.rand(*s, device=DEV, generator=g)  # noqa: E731
    randn = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    n, scene = case["points"], case["scene"]
    if scene == "near":
        means = torch.cat([2 * rand(n, 2) - 1, 2 + 2 * rand(n, 1)], 1)
        lo, hi = 0.05, 0.5
    else:
        means = 6 * rand(n, 3) - 3
        lo, hi = 0.005, 0.05
        if scene == "clusters":
            means = means[:64][torch.randint(min(64, n), (n,), device=DEV, generator=g)] + 0.3 * randn(n, 3)
    s2 = torch.exp(math.log(lo) + math.log(hi / lo) * rand(n, 2))
    q = randn(n, 4)
    q = q / q.norm(dim=-1, keepdim=True)
    logit = randn(n, 1)
    deg = case.get("sh_degree", 0)
    sh = rand(n, (deg + 1) ** 2, 3) if scene == "near" else 0.2 * randn(n, (deg + 1) ** 2, 3)
    if scene != "near":
        sh[:, 0] += 1.2
    texels, side = case.get("texels", 0), case.get("side", 1)
    if texels:
        size = s2.prod(-1) / (means[:, 2] ** 2 if scene == "near" else 64.0)
        hw = torch.sqrt(texels * size / size.sum()).floor().clamp(2, 16).int()
        rows = texels + 4 * n
    else:
        hw = torch.full((n,), side, dtype=torch.int32, device=DEV)
        rows = side * side * n
    dims = torch.stack([hw, hw, ((hw * hw).cumsum(0) - hw * hw).int()], -1).int().contiguous()
    ax1, ax2, _ = _axes(q)
    return dict(means=means, scales=torch.cat([s2, 1e-5 * s2.mean(-1, keepdim=True)], -1), quats=q,
                opacity=torch.sigmoid(logit), logit=logit, sh_coeffs=sh, uv0=torch.full((n, 1, 2), 0.5, device=DEV),
                umap=(ax1 / (6 * s2[:, :1]))[:, None].contiguous(), vmap=(ax2 / (6 * s2[:, 1:]))[:, None].contiguous(),
                texture_dims=dims, texture=rand(rows, 3))


def _bf16x4(tex):
    out = torch.zeros(tex.shape[0], 4, dtype=torch.bfloat16, device=tex.device)
    out[:, :3] = tex
    return out


PARAMS = ("opacity", "means", "scales", "quats", "uv0", "umap", "vmap", "texture", "sh_coeffs")


def _raw(s):
    """The trainer's parameters of a scene: log-scales, unnormalised quaternions, chart mapping, opacity logits."""
    scale = s["scales"].clone()
    n = scale.shape[0]
    theta = torch.atan2(s["means"][:, 0], s["means"][:, 1])
    uvs = -torch.log(6 * scale[:, :2].mean(-1))
    mapping = torch.stack([torch.full((n,), 0.5, device=DEV), torch.full((n,), 0.5, device=DEV), uvs, theta], -1)
    return dict(raw_scales=scale.log(), raw_quats=s["quats"] * (0.5 + s["opacity"]), mapping=mapping[:, None].contiguous(),
                raw_opacity=s["logit"][:, 0].contiguous())


def prepare(case, seed):
    kind = case["kind"]
    r = random.Random(seed)
    g = torch.Generator(device=DEV).manual_seed(seed + 1000003)
    rand = lambda *s: torch.rand(*s, device=DEV, generator=g)  # noqa: E731
    randn = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    st = dict(case=case)
    if kind == "sample":
        m, side, q, c = case["charts"], case["side"], case["queries"], case["channels"]
        h = torch.randint(1, side + 1, (m, 2), device=DEV, generator=g).int()
        dims = torch.cat([h, (torch.arange(m, device=DEV) * side * side).int()[:, None]], 1)
        at = torch.randint(m, (q,), device=DEV, generator=g)
        st.update(dims=dims[at].contiguous(), tex=rand(m * side * side, c).requires_grad_(),
                  uvs=(1.1 * rand(q, 2) - 0.05).requires_grad_(), info=(q, 1, c), up=randn(q, c))
        return st
    if kind == "params":
        n = case["points"]
        s = _scene(dict(case, scene="cube"), seed)
        st.update({k: v.requires_grad_() for k, v in _raw(s).items()}, sh=s["sh_coeffs"].requires_grad_(),
                  dirs=s["means"] - torch.tensor([0.0, 0.0, -8.0], device=DEV),
                  ups=[randn(n, 3), randn(n, 4), randn(n, 1, 2), randn(n, 1, 3), randn(n, 1, 3), randn(n, 1),
                       randn(n, 3)])
        return st
    s = _scene(case, seed)
    cams = [_camera(case["scene"], w, h, r) for w, h in _sizes(case)]
    st.update(scene=s)
    if kind == "edit":
        w, h = case["width"], case["height"]
        vm = cams[0][0]
        mid = 3.0 if case["scene"] == "near" else 8.0
        st.update(vm=vm.float().to(DEV), c2w=torch.linalg.inv(vm).float().to(DEV), intr=cams[0][1:],
                  img=rand(h, w, 3), alpha=(rand(h, w, 1) > 0.3).float(), lower=mid - 2 * rand(h, w),
                  upper=mid + 2 * rand(h, w))
        return st
    if case.get("bf16"):
        s["texture"] = _bf16x4(s["texture"])
    if kind == "view":
        w, h = case["width"], case["height"]
        vm = cams[0][0]
        st.update(vm=vm.float().to(DEV), c2w=torch.linalg.inv(vm).float().to(DEV), intr=cams[0][1:],
                  info=(s["means"].shape[0], 1, 3), bg=torch.zeros(3, device=DEV))
        if case["grad"]:
            for k in PARAMS:
                s[k].requires_grad_()
            p = float(w * h)  # what a mean over the picture's pixels hands back
            st["ups"] = [randn(h, w, 3) / p, torch.full((h, w), LOSS["reg"] / p, device=DEV), randn(h, w, 3) / p,
                         0.1 * randn(h, w, 3) / p]
        return st
    # kind == "batch"
    cams = [B.Camera(vm.float(), fx, fy, cx, cy, w, h) for (vm, fx, fy, cx, cy), (w, h) in zip(cams, _sizes(case))]
    if case["bf16"]:
        s["sh_coeffs"] = s["sh_coeffs"].bfloat16()
    deg = case["sh_degree"]
    if case["raw"]:
        raw = _raw(s)
        st["obj"] = B.RawScene(means=s["means"], sh_coeffs=s["sh_coeffs"], sh_degree=deg,
                               texture_dims=s["texture_dims"], texture=s["texture"], **raw)
    else:
        st["obj"] = B.Scene(means=s["means"], scales=s["scales"], quats=s["quats"], opacity=s["opacity"],
                            sh_coeffs=s["sh_coeffs"], sh_degree=deg, uv0=s["uv0"], umap=s["umap"], vmap=s["vmap"],
                            texture_dims=s["texture_dims"], texture=s["texture"])
    st["cams"] = cams
    R = B.BatchRenderer(cams, case["points"], texture_dtype=s["texture"].dtype, block_width=case["block_width"],
                        settings=SETTINGS, bwd_ctas=case["ctas"], loss_weights=LOSS, device=DEV)
    for _ in range(3):  # size the intersection buffers, as the benchmark does
        (R.bin_raw if case["raw"] else R.bin)(st["obj"])
        if R.check_capacity():
            break
        R.grow(1.25)
    st["R"] = R
    if case["grad"]:
        st["tgt"] = (rand(R.total_pixels, 3), rand(R.total_pixels, 3))
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _view_inputs(st, w, h):
    s = st["scene"]
    means = s["means"].detach()
    centers, extents = get_aabb_2d(means, s["scales"].detach(), 1.0, s["quats"].detach(), st["vm"], st["intr"])
    _, depths = project_points(means, st["vm"], st["intr"])
    return centers, extents, depths, get_num_tiles_hit_2d(centers, extents, h, w, 16)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "sample":
        out = texture_sample(st["info"], st["dims"], st["tex"], st["uvs"])
        v_tex, v_uvs = torch.autograd.grad(out, (st["tex"], st["uvs"]), st["up"])
        return dict(out=out.detach(), v_texture=v_tex, v_uvs=v_uvs)
    if kind == "params":
        ins = [st[k] for k in ("raw_scales", "raw_quats", "mapping", "raw_opacity")]
        outs = list(preprocess(*ins)) + [spherical_harmonics(case["sh_degree"], st["dirs"], st["sh"])]
        grads = torch.autograd.grad(outs, ins + [st["sh"]], st["ups"])
        return dict(outs=[o.detach() for o in outs], grads=list(grads))
    if kind == "edit":
        s, w, h = st["scene"], case["width"], case["height"]
        centers, extents, depths, hits = _view_inputs(st, w, h)
        return texture_edit((case["points"], 1, 5), s["texture_dims"], st["img"], st["alpha"], st["lower"],
                            st["upper"], centers, extents, depths, hits, s["opacity"], s["means"], s["scales"], 1.0,
                            s["quats"], s["uv0"], s["umap"], s["vmap"], st["vm"], st["c2w"], *st["intr"], h, w, 16, 0)
    if kind == "view":
        s, w, h = st["scene"], case["width"], case["height"]
        colors = spherical_harmonics(case["sh_degree"], s["means"].detach() - st["c2w"][:3, 3], s["sh_coeffs"])
        outs = texture_gaussians(st["info"], s["texture_dims"], *_view_inputs(st, w, h), colors, s["opacity"],
                                 s["means"], s["scales"], 1.0, s["quats"], s["uv0"], s["umap"], s["vmap"],
                                 s["texture"], st["vm"], st["c2w"], *st["intr"], h, w, 16, SETTINGS, st["bg"])
        img, depth, reg, alpha, tex, normal = outs
        res = dict(img=img.detach(), depth=depth.detach(), reg=reg.detach(), alpha=alpha.detach(), tex=tex.detach(),
                   normal=normal.detach())
        if case["grad"]:
            grads = torch.autograd.grad((img, reg, tex, normal), [s[k] for k in PARAMS], st["ups"])
            res.update({"v_" + k: v for k, v in zip(PARAMS, grads)})
        return res
    R, obj = st["R"], st["obj"]
    res = {}
    if not case["grad"]:
        R.forward(R.bin_raw(obj) if case["raw"] else _binned(R, obj))
    elif case["raw"]:
        res["loss"] = R.step_raw(obj, *st["tgt"])
        res.update({"v_" + k: v for k, v in R.raw_grads.items()})
    else:
        res["loss"] = R.step(obj, *st["tgt"])
        res.update({"v_" + k: v for k, v in R.grads.items()})
    res.update({k: R.out[k] for k in ("img", "depth", "reg", "texture", "normal", "final_T")})
    return res


def _binned(R, obj):
    R.bin(obj)
    return obj


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: every parameter, texel and upstream gradient read once, every
    output and gradient written once.  Operations: about 18 splats contribute
    to a covered pixel before it saturates; each costs about 90 operations
    forward and 300 backward (ray-plane solve, exp, bilinear lookup, blend and
    their adjoints)."""
    kind = case["kind"]
    if kind == "sample":
        q, c = case["queries"], case["channels"]
        texels = min(case["charts"] * case["side"] ** 2, 4 * q)
        return dict(bytes=4.0 * (q * (3 + 2 + c + c + 2) + 2 * texels * c), flops=q * (20.0 + 30.0 * c))
    nb = (case.get("sh_degree", 0) + 1) ** 2
    n = case["points"]
    if kind == "params":
        return dict(bytes=4.0 * n * (2 * (3 + 4 + 4 + 1) + 2 * (3 + 4 + 2 + 3 + 3 + 1) + 2 * (3 * nb + 3) + 3),
                    flops=n * (400.0 + 12.0 * nb))
    pix = float(sum(w * h for w, h in _sizes(case)))
    if kind == "edit":
        return dict(bytes=4.0 * (n * 22 + pix * 6 + 5 * n * case["side"] ** 2), flops=pix * 18 * 90)
    texels = case["texels"] + 4 * n if case["texels"] else n
    tb, sb = (8, 2 if kind == "batch" else 4) if case.get("bf16") else (12, 4)
    b = n * (22 * 4 + 3 * nb * sb) + texels * tb + pix * 12 * 4
    if case["grad"]:
        b += n * (19 + 3 * nb) * 4 + texels * (16 if case.get("bf16") else 12) + pix * 10 * 4
    return dict(bytes=float(b), flops=pix * 18 * (390.0 if case["grad"] else 90.0))


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _sh_basis(deg, d):
    x, y, z = (d / d.norm(dim=-1, keepdim=True)).unbind(-1)
    Y = [torch.full_like(x, 0.28209479177387814)]
    if deg > 0:
        Y += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if deg > 1:
        Y += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
              0.31539156525252005 * (2 * z * z - x * x - y * y), -1.0925484305920792 * x * z,
              0.5462742152960396 * (x * x - y * y)]
    if deg > 2:
        Y += [-0.5900435899266435 * y * (3 * x * x - y * y), 2.890611442640554 * x * y * z,
              -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
              0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
              -0.4570457994644658 * x * (4 * z * z - x * x - y * y), 1.445305721320277 * z * (x * x - y * y),
              -0.5900435899266435 * x * (x * x - 3 * y * y)]
    return torch.stack(Y, -1)


def _tiles(p, cam, w, h, bw):
    """Per tile the Gaussians whose +-3 sigma box meets it, front to back: (ids, first, count)."""
    vm, fx, fy, cx, cy = cam
    R, t = vm[:3, :3], vm[:3, 3]
    ax1, ax2, _ = _axes(p["quats"])
    z = (p["means"] @ R.T + t)[:, 2]
    pix = []
    for a in (3, -3):
        for b in (3, -3):
            c = (p["means"] + a * p["scales"][:, :1] * ax1 + b * p["scales"][:, 1:2] * ax2) @ R.T + t
            rz = 1 / (c[:, 2].clamp(min=0.01) + 1e-6)
            pix.append(torch.stack([c[:, 0] * rz * fx + cx, c[:, 1] * rz * fy + cy], -1))
    pix = torch.stack(pix)
    lo, hi = pix.amin(0) / bw, pix.amax(0) / bw
    n = torch.tensor([(w + bw - 1) // bw, (h + bw - 1) // bw], device=DEV)
    t0 = torch.minimum(lo.trunc().long().clamp(min=0), n)
    t1 = torch.minimum((hi + 1).trunc().long().clamp(min=0), n)
    t1[z <= 0.01] = t0[z <= 0.01]
    span = (t1 - t0).clamp(min=0)
    cnt = span.prod(-1)
    gid = torch.repeat_interleave(torch.arange(cnt.shape[0], device=DEV), cnt)
    k = torch.arange(gid.shape[0], device=DEV) - (cnt.cumsum(0) - cnt)[gid]
    tile = (t0[gid, 1] + k // span[gid, 0]) * n[0] + t0[gid, 0] + k % span[gid, 0]
    order = torch.argsort(z[gid], stable=True)
    order = order[torch.argsort(tile[order], stable=True)]
    count = torch.bincount(tile, minlength=int(n[0] * n[1]))
    return gid[order], count.cumsum(0) - count, count


def _through(x, y):
    """y's value, x's gradient."""
    return x + (y - x).detach()


def _render(p, colors, cam, w, h, bw, each, most=24_000_000):
    """Composites one view chunk by chunk of tiles; ``each(pix, keep, outs, pairs)``
    gets the chunk's pixel indices [tiles, bw^2] (in the picture where ``keep``),
    the outputs of the kept pixels and the chunk's (splat, pixel) pairs.  Returns
    False if there are too many pairs to finish in time."""
    vm, fx, fy, cx, cy = cam
    R = vm[:3, :3]
    with torch.no_grad():
        ids, first, count = _tiles(p, cam, w, h, bw)
    if ids.shape[0] * bw * bw > 1.2e9:
        return False
    tx = (w + bw - 1) // bw
    by = torch.argsort(count)
    lens = count[by].tolist()
    loc = torch.arange(bw * bw, device=DEV)
    at, end = 0, len(lens)
    while at < end:
        to = at + 1
        while to < end and (to + 1 - at) * max(1, lens[to]) * bw * bw <= most:
            to += 1
        tiles, L = by[at:to], max(1, lens[to - 1])
        at = to
        py, px = (tiles // tx)[:, None] * bw + loc // bw, (tiles % tx)[:, None] * bw + loc % bw
        keep = (px < w) & (py < h)
        k = torch.arange(L, device=DEV)
        live = k[None] < count[tiles][:, None]
        gid = ids[(first[tiles][:, None] + k).clamp(max=max(ids.shape[0] - 1, 0))] if ids.shape[0] else torch.zeros_like(k)[None].expand(len(tiles), L)
        u, v = (px.double() + 0.5 - cx) / fx, (py.double() + 0.5 - cy) / fy
        d = torch.stack([u, v, torch.ones_like(u)], -1)
        idn = 1 / d.norm(dim=-1)
        ray = (d * idn[..., None]) @ R  # world
        eye = -R.T @ vm[:3, 3]
        G = {n: x[gid] for n, x in p.items() if n not in ("texture", "texture_dims", "uv0", "umap", "vmap")}
        uv0, um, vv = p["uv0"][:, 0][gid], p["umap"][:, 0][gid], p["vmap"][:, 0][gid]
        a1, a2, a3 = _axes(G["quats"])
        rel = G["means"] - eye
        dot = lambda x: torch.einsum("tlc,tpc->tlp", x, ray)  # noqa: E731
        den = dot(a3)
        den = torch.where((den >= 0) & (den < 1e-6), torch.full_like(den, 1e-6),
                          torch.where((den <= 0) & (den > -1e-6), torch.full_like(den, -1e-6), den))
        t = (a3 * rel).sum(-1)[..., None] / den
        on = lambda x: dot(x) * t - (x * rel).sum(-1)[..., None]  # noqa: E731  (x . (hit - mean))
        l1, l2 = on(a1) / G["scales"][..., :1], on(a2) / G["scales"][..., 1:2]
        raw = G["opacity"][..., :1] * torch.exp(-0.5 * (l1 * l1 + l2 * l2))
        alpha = _through(raw, raw.clamp(max=0.99))
        with torch.no_grad():
            ok = live[..., None] & (t >= 0.01) & (t <= 1000) & (alpha >= 1 / 255.0)
            T0 = torch.where(ok, 1 - alpha, torch.ones_like(alpha)).cumprod(1)
            T0 = torch.cat([torch.ones_like(T0[:, :1]), T0[:, :-1]], 1)
            stop = live[..., None] & (T0 * (1 - alpha) <= 1e-4)
            ok &= ~(stop.cumsum(1) > 0)
        al = torch.where(ok, alpha, torch.zeros_like(alpha))
        Tn = (1 - al).cumprod(1)
        T = torch.cat([torch.ones_like(Tn[:, :1]), Tn[:, :-1]], 1)
        vis = al * T
        t = torch.where(ok, t, torch.zeros_like(t))
        tu, tv = uv0[..., :1] + on(um), uv0[..., 1:] + on(vv)
        dims = p["texture_dims"][gid].long()
        hh, ww, start = dims[..., :1], dims[..., 1:2], dims[..., 2:]
        fu, fv = _through(tu, tu.clamp(0, 1)) * hh, _through(tv, tv.clamp(0, 1)) * ww
        iu, iv = fu.detach().trunc().long(), fv.detach().trunc().long()
        ru, rv = fu - iu, fv - iv
        iu1, iv1 = torch.minimum(iu + 1, hh - 1), torch.minimum(iv + 1, ww - 1)
        iu, iv = torch.minimum(iu, hh - 1), torch.minimum(iv, ww - 1)
        rows = [(start + i * ww + j) for i in (iu, iu1) for j in (iv, iv1)]
        wts = [a * b for a in (1 - ru, ru) for b in (1 - rv, rv)]
        pairs = dict(ok=ok, rows=rows, wts=wts, tz=t * idn[:, None])
        if colors is None:
            outs = None
        else:
            tex = 0
            for q in range(4):
                texel = p["texture"][rows[q]]
                tex = tex + torch.einsum("tlp,tlpc->tpc", vis * wts[q], texel)
            S0, S1, S2 = vis.cumsum(1) - vis, (vis * t).cumsum(1) - vis * t, (vis * t * t).cumsum(1) - vis * t * t
            half = ok & (T.detach() > 0.5)
            last = (half * (k[None, :, None] + 1)).amax(1, keepdim=True)
            depth = torch.where(last[:, 0] > 0, (t * idn[:, None]).gather(1, (last - 1).clamp(min=0))[:, 0],
                                torch.zeros_like(idn))
            outs = dict(img=torch.einsum("tlp,tlc->tpc", vis, colors[gid]), depth=depth,
                        reg=(vis * (t * t * S0 + S2 - 2 * t * S1)).sum(1), final_T=Tn[:, -1],
                        texture=tex, normal=torch.einsum("tlp,tlc->tpc", vis, a3))
            outs = {n: x[keep] for n, x in outs.items()}
        each(py * w + px, keep, outs, pairs)
    return True


def _exact_views(case, p, sh, views, bw, grad_of):
    """Outputs of all views, and the gradients of the sum of ``grad_of(v, pixels, outs)`` w.r.t. p, sh and
    the views' colours."""
    deg = case["sh_degree"]
    leaves = {k: x.clone().requires_grad_(x.is_floating_point() and grad_of is not None) for k, x in p.items()}
    sizes = _sizes(case)
    outs, v_sh, v_cols, loss = [], torch.zeros_like(sh), [], 0.0
    for v, ((w, h), cam) in enumerate(zip(sizes, views)):
        eye = -cam[0][:3, :3].T @ cam[0][:3, 3]
        Y = _sh_basis(deg, p["means"] - eye)
        colors = torch.einsum("nb,nbc->nc", Y, sh).requires_grad_(grad_of is not None)
        full = {}
        box = [0.0]

        def each(pix, keep, o, _):
            pixels = pix[keep]
            for k, x in o.items():
                if k not in full:
                    full[k] = torch.zeros((h * w,) + tuple(x.shape[1:]), dtype=torch.float64, device=DEV)
                full[k][pixels] = x.detach()
            if grad_of is not None:
                part = grad_of(v, pixels, o)
                box[0] += float(part.detach())
                if part.requires_grad:
                    part.backward()

        with torch.set_grad_enabled(grad_of is not None):
            if not _render(leaves, colors, cam, w, h, bw, each):
                return None
        loss += box[0]
        outs.append(full)
        if grad_of is not None:
            vc = colors.grad if colors.grad is not None else torch.zeros_like(colors)
            v_cols.append(vc)
            v_sh += Y[:, :, None] * vc[:, None, :]
    grads = {k: (x.grad if x.grad is not None else torch.zeros_like(x)) for k, x in leaves.items() if x.requires_grad}
    grads["sh_coeffs"] = v_sh
    return loss, outs, grads, v_cols


def exact(case, seed):
    kind = case["kind"]
    st = prepare(case, seed)
    if kind == "sample":
        tex = st["tex"].detach().double().requires_grad_()
        uvs = st["uvs"].detach().double().requires_grad_()
        d = st["dims"].long()
        f = uvs.clamp(0, 1) * d[:, :2]
        i = f.detach().trunc().long()
        r = f - i
        i1 = torch.minimum(i + 1, d[:, :2] - 1)
        i = torch.minimum(i, d[:, :2] - 1)
        out = 0
        for a, wa in ((i, 1 - r), (i1, r)):
            for b, wb in ((i, 1 - r), (i1, r)):
                out = out + (wa[:, 0] * wb[:, 1])[:, None] * tex[d[:, 2] + a[:, 0] * d[:, 1] + b[:, 1]]
        v_tex, v_uvs = torch.autograd.grad(out, (tex, uvs), st["up"].double())
        return dict(out=out.detach(), v_texture=v_tex, v_uvs=v_uvs)
    if kind == "params":
        raw = [st[k].detach().double().requires_grad_() for k in ("raw_scales", "raw_quats", "mapping", "raw_opacity")]
        sh = st["sh"].detach().double().requires_grad_()
        outs = _activate(*raw)
        outs = list(outs) + [torch.einsum("nb,nbc->nc", _sh_basis(case["sh_degree"], st["dirs"].double()), sh)]
        # the third scale follows the other two and hands nothing back
        ups = [u.double() for u in st["ups"]]
        ups[0] = ups[0] * torch.tensor([1.0, 1.0, 0.0], device=DEV, dtype=torch.float64)
        grads = torch.autograd.grad(outs, raw + [sh], ups)
        return dict(outs=[o.detach() for o in outs], grads=list(grads))
    r = random.Random(seed)
    views = []
    for w, h in _sizes(case):
        vm, *intr = _camera(case["scene"], w, h, r)
        views.append((vm.float().double().to(DEV), *intr))
    s = {k: (x.detach().double() if x.is_floating_point() else x) for k, x in st["scene"].items()}
    if s["texture"].shape[1] == 4:
        s["texture"] = s["texture"][:, :3].contiguous()
    names = ("means", "scales", "quats", "opacity", "uv0", "umap", "vmap", "texture", "texture_dims")
    if kind == "edit":
        w, h = case["width"], case["height"]
        total = case["side"] ** 2 * case["points"]
        out = torch.zeros(total, 5, dtype=torch.float64, device=DEV)
        a = st["alpha"].double().reshape(-1)
        val = torch.cat([st["img"].double().reshape(-1, 3) * a[:, None], a[:, None], torch.ones_like(a)[:, None]], 1)
        lo, hi = st["lower"].double().reshape(-1), st["upper"].double().reshape(-1)

        def each(pix, keep, _, q):
            at = torch.where(keep, pix, torch.zeros_like(pix))
            use = q["ok"] & keep[:, None] & (q["tz"] >= lo[at][:, None]) & (q["tz"] <= hi[at][:, None])
            where = use.nonzero(as_tuple=True)
            src = val[at[where[0], where[2]]]
            for rows, wt in zip(q["rows"], q["wts"]):
                out.index_add_(0, rows[where], wt[where][:, None] * src)

        with torch.no_grad():
            return out if _render({k: s[k] for k in names}, None, views[0], w, h, 16, each) else None
    if kind == "view":
        w, h = case["width"], case["height"]
        p = {k: s[k] for k in names}
        ups = [u.double().reshape((h * w,) + tuple(u.shape[2:])) for u in st["ups"]] if case["grad"] else None

        def grad_of(v, pix, o):
            return sum((x * u[pix]).sum() for x, u in zip((o["img"], o["reg"], o["texture"], o["normal"]), ups))

        got = _exact_views(case, p, s["sh_coeffs"], views, 16, grad_of if case["grad"] else None)
        if got is None:
            return None
        o = got[1][0]
        sq = lambda x: x.reshape((h, w) + tuple(x.shape[1:]))  # noqa: E731
        res = dict(img=sq(o["img"]), depth=sq(o["depth"]), reg=sq(o["reg"]), alpha=sq(1 - o["final_T"]),
                   tex=sq(o["texture"]), normal=sq(o["normal"]))
        if case["grad"]:
            res.update({"v_" + k: got[2][k] for k in PARAMS})
        return res
    # kind == "batch"
    p = {k: s[k] for k in names if k in s}
    raw = None
    if case["raw"]:
        obj = st["obj"]
        raw = [getattr(obj, k).double().requires_grad_() for k in ("raw_scales", "raw_quats", "mapping", "raw_opacity")]
        act = _activate(*raw)
        p.update({k: x.detach() for k, x in zip(("scales", "quats", "uv0", "umap", "vmap", "opacity"), act)})
    off = [0]
    for w, h in _sizes(case):
        off.append(off[-1] + w * h)
    grad_of = None
    if case["grad"]:
        ti, tt = (x.double() for x in st["tgt"])

        def grad_of(v, pix, o):
            inv, at = 1.0 / (off[v + 1] - off[v]), off[v] + pix
            n = o["normal"]
            return inv * (LOSS["img"] / 3 * ((o["img"] - ti[at]) ** 2).sum()
                          + LOSS["texture"] / 3 * ((o["texture"] - tt[at]) ** 2).sum() + LOSS["reg"] * o["reg"].sum()
                          + LOSS["normal"] * (n[:, 0] ** 2 + n[:, 1] ** 2 + (1 - n[:, 2]) ** 2).sum())

    if sum(w * h for w, h in _sizes(case)) * (case["points"] / 1e5) > 4e6:
        return None
    got = _exact_views(case, p, s["sh_coeffs"], views, case["block_width"], grad_of)
    if got is None:
        return None
    loss, outs, grads, v_cols = got
    res = {k: torch.cat([o[k] for o in outs]) for k in ("img", "depth", "reg", "texture", "normal", "final_T")}
    if case["grad"]:
        res["loss"] = torch.tensor([loss], dtype=torch.float64)
        pad4 = lambda x: torch.cat([x, torch.zeros_like(x[..., :1])], -1)  # noqa: E731
        res["v_vcolors"] = pad4(torch.stack(v_cols))
        if case["bf16"]:
            grads["texture"] = pad4(grads["texture"])
        if raw is not None:
            back = torch.autograd.grad(act, raw, [grads[k] for k in ("scales", "quats", "uv0", "umap", "vmap",
                                                                     "opacity")])
            for k, x in zip(("raw_scales", "raw_quats", "mapping", "raw_opacity"), back):
                res["v_" + k] = x
            for k in ("means", "texture", "sh_coeffs"):
                res["v_" + k] = grads[k]
        else:
            res.update({"v_" + k: grads[k] for k in PARAMS})
    return res


def _activate(raw_scales, raw_quats, mapping, raw_opacity):
    s2 = raw_scales[:, :2].exp()
    scales = torch.cat([s2, 1e-5 * s2.mean(-1, keepdim=True)], -1)
    q = raw_quats / raw_quats.norm(dim=-1, keepdim=True)
    a1, a2, _ = _axes(q)
    us, th = mapping[..., 2:3].exp(), mapping[..., 3:4]
    um = us * (a1[:, None] * th.cos() + a2[:, None] * th.sin())
    vm = us * (a2[:, None] * th.cos() - a1[:, None] * th.sin())
    return scales, q, mapping[..., :2], um, vm, torch.sigmoid(raw_opacity).reshape(-1, 1)

