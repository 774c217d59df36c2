"""The work that a program built on this package has it do, as cases that can be timed and checked.

Each case is one call of a public entry point, at a size that its users run:

* ``render``: ``Microfacet.eval`` of one or more materials, alone (a preview, a saved re-render) or with the
  gradient that a loss hands back (``torch.autograd``): the building block of the reference's own loops;
* ``optim``: ``SvbrdfOptim.optim``, the per-pixel fit of one material, with a fixed or a learnt light;
* ``batch``: ``BatchedOptim.run``, many materials of uneven size fitted together;
* ``descriptor``: ``VGGDescriptor.loss_and_grad``, the feature (and Gram) loss with its gradient;
* ``layer``: one style layer of the generator, forward and backward;
* ``latent``: the gradient of the image loss with respect to the W+ latent and the noise maps, through generator and
  renderer. (The loop's own step follows with a fresh Adam, whose update is lr times the gradient's sign: the gradient
  is what can be compared.)
* ``envmap``: one frame of the novel-view video.

``listed`` names the fixed cases, ``draw`` gives more of the same ranges, ``prepare`` makes what the program has in hand
before the call, ``run`` is the call, ``work`` what it cannot do without, and ``exact`` the same result in 64 bits.
"""
import importlib
import math
from types import SimpleNamespace

import numpy as np
import torch
import torch.nn.functional as Fn

gb = importlib.import_module("svbrdf-diff-renderer_gb300")

DEV = torch.device("cuda:0")
SIZE_CM = gb.scenes.GRID_SIZE_CM
LIGHT = gb.scenes.LIGHT_POW
EPS = 1e-6
# arithmetic of one texel under one view: forward render, and with the adjoint (transcendentals counted as one each)
FLOPS_VIEW_FWD, FLOPS_VIEW_STEP = 90, 230


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a preview of a small material: the shortest call, launch and host latency
        {"name": "render_preview_128", "kind": "render", "res": 128, "views": 9, "batch": 1, "grad": False, "coloc": True,
         "light": False},
        # a capture whose lights stand apart from the cameras, an odd crop, the light's gradient asked for
        {"name": "render_grad_general_333", "kind": "render", "res": 333, "views": 5, "batch": 1, "grad": True,
         "coloc": False, "light": True},
        # the reference's nine flash photos at full resolution: one forward and backward of the plain loop
        {"name": "render_grad_1024", "kind": "render", "res": 1024, "views": 9, "batch": 1, "grad": True, "coloc": True,
         "light": False},
        # the reference's own per-pixel fit: 256^2, nine photos, MSE, a short call
        {"name": "optim_256", "kind": "optim", "res": 256, "views": 9, "epochs": 20, "loss": "mse", "light": False},
        # a fit that learns the flash's power too: every epoch ends in a reduction over the whole material
        {"name": "optim_light_512", "kind": "optim", "res": 512, "views": 9, "epochs": 50, "loss": "log1p", "light": True},
        # a shelf of captures fitted together: resolutions 256..1024, 5..16 photos each
        {"name": "batch_uneven_32", "kind": "batch", "materials": 32, "lo": 256, "hi": 1024, "vmin": 5, "vmax": 16,
         "iters": 50, "loss": "log1p"},
        # feature and Gram loss of nine 512^2 renders
        {"name": "descriptor_512", "kind": "descriptor", "mode": "config", "views": 9, "h": 512, "w": 512},
        # the reference's own feature loss (average pools, to relu4_2) of nine 256^2 renders
        {"name": "descriptor_reference_256", "kind": "descriptor", "mode": "reference", "views": 9, "h": 256, "w": 256},
        # an ordinary up-sampling layer of the generator
        {"name": "layer_up_128", "kind": "layer", "up": True, "res": 128, "batch": 4},
        # the generator's last convolution, the one with the largest maps
        {"name": "layer_conv_256", "kind": "layer", "up": False, "res": 256, "batch": 8},
        # the latent fit of a batch of materials
        {"name": "latent_grad_16", "kind": "latent", "batch": 16, "views": 9},
        # a frame of the novel-view video
        {"name": "envmap_frame_256", "kind": "envmap", "res": 256, "tex": 256, "spp": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "optim", "batch", "descriptor", "layer", "latent", "envmap"])
    if kind == "render":
        res, views, batch = _log(rng, 48, 1024), rng.randint(1, 16), rng.choice([1, 1, 2, 4, 9])
        while res * res * views * batch > 1024 * 1024 * 9:
            res = res * 3 // 4
        grad = rng.random() < 0.7
        return {"kind": kind, "res": res, "views": views, "batch": batch, "grad": grad, "coloc": rng.random() < 0.7,
                "light": grad and rng.random() < 0.4}
    if kind == "optim":
        return {"kind": kind, "res": _log(rng, 64, 1024), "views": rng.randint(3, 16), "epochs": _log(rng, 5, 50),
                "loss": rng.choice(["mse", "log1p"]), "light": rng.random() < 0.3}
    if kind == "batch":
        lo = _log(rng, 64, 384)
        return {"kind": kind, "materials": _log(rng, 2, 24), "lo": lo, "hi": min(1024, lo * rng.randint(1, 4)),
                "vmin": rng.randint(3, 6), "vmax": rng.randint(7, 16), "iters": _log(rng, 5, 50),
                "loss": rng.choice(["mse", "log1p"])}
    if kind == "descriptor":
        mode = rng.choice(["config", "reference"])
        step, top = (32, 512) if mode == "config" else (16, 256)
        side = lambda: max(4, min(top // step, round(_log(rng, 64, top) / step))) * step
        return {"kind": kind, "mode": mode, "views": rng.randint(1, 9), "h": side(), "w": side()}
    if kind == "layer":
        res = rng.choice([8, 16, 32, 64, 128, 256])
        return {"kind": kind, "up": rng.random() < 0.5, "res": res, "batch": rng.randint(1, 8 if res == 256 else 16)}
    if kind == "latent":
        return {"kind": kind, "batch": rng.randint(1, 15), "views": rng.randint(3, 9)}
    return {"kind": kind, "res": _log(rng, 64, 256), "tex": _log(rng, 64, 1024), "spp": _log(rng, 16, 256)}


# ------------------------------------------------------------------------------------------------ inputs
def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(seed * 1000003 + 17)


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _material(res, g):
    """[1, 9, res, res] smooth seeded maps in [-1, 1], of the ranges of ``scenes.make_material``: noise blurred by 4
    texels, normals from a height field that tilts 30 degrees at most."""
    f = gb.scenes.smooth_field(torch.randn(8, res, res, generator=g, device=DEV)) if res >= 26 else torch.randn(
        8, res, res, generator=g, device=DEV)
    lo, hi = f.amin((1, 2), keepdim=True), f.amax((1, 2), keepdim=True)
    f = (f - lo) / (hi - lo)
    dif, spe, rgh = 0.05 + 0.85 * f[0:3], 0.02 + 0.48 * f[3:6], 0.1 + 0.8 * f[6:7]
    dx, dy = torch.roll(f[7], -1, 1) - torch.roll(f[7], 1, 1), torch.roll(f[7], -1, 0) - torch.roll(f[7], 1, 0)
    k = math.tan(math.radians(30.0)) / (dx * dx + dy * dy).max().sqrt()
    inv = torch.rsqrt((dx * dx + dy * dy) * k * k + 1.0)
    return torch.cat((dif * 2 - 1, (-dx * k * inv)[None], (-dy * k * inv)[None], rgh * 2 - 1, spe * 2 - 1))[None].contiguous()


def _views(n, g, coloc=True):
    """Camera and light positions [n, 3] in cm: flashes within +-8 cm at 25 to 35 cm, as the batched workload has them."""
    def points():
        return torch.cat(((_uniform(g, n, 2) * 2 - 1) * 8.0, 25.0 + 10.0 * _uniform(g, n, 1)), 1)

    cam = points()
    return cam, (cam.clone() if coloc else points())


def _light():
    return torch.full((3,), LIGHT, device=DEV)


def _photos(tex, cam, lit, g):
    """What was photographed: the material's renders with noise, clamped to [0, 1]."""
    with torch.no_grad():
        r = gb.Microfacet(tex.shape[-1], cam.shape[0], SIZE_CM, [cam, lit, _light()], DEV).eval(tex)
        return (r + 0.01 * torch.randn(r.shape, generator=g, device=DEV)).clamp(0, 1).contiguous()


def _capture(res, views, g):
    gt = _material(res, g)
    cam, lit = _views(views, g)
    return gb.scenes.Scene(res=res, size=SIZE_CM, camera_pos=cam, light_pos=lit, light_pow=_light(), gt=gt,
                           targets=_photos(gt, cam, lit, g), init=gb.scenes.const_init(res, device=DEV))


def _batch_shapes(case, seed):
    """(resolution, views) of a batch's materials: even sizes between lo and hi, as cropped and scaled photos have. The
    shapes are the case's own; the seed changes what the materials are."""
    r = np.random.RandomState(case["materials"] * 7919 + case["lo"])
    if (case["lo"], case["hi"]) == (256, 1024):
        sides = r.choice([256, 512, 1024], case["materials"])
    else:
        sides = [2 * int(round(x / 2)) for x in np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"] + 1e-9),
                                                                case["materials"]))]
    return [(int(s), int(v)) for s, v in zip(sides, r.randint(case["vmin"], case["vmax"] + 1, case["materials"]))]


_GENERATOR = []


def _generator():
    """The one generator of the program: 256^2, 9 channels, seeded weights; noise strengths and biases as a trained one
    has them, not zero."""
    if not _GENERATOR:
        gen = gb.materialgan.StyleGAN2Generator(256, seed=0)
        g = torch.Generator().manual_seed(5)
        with torch.no_grad():
            for m in [gen.conv4, *gen.ups, *gen.convs]:
                m.noise_strength.fill_(0.05 + 0.1 * float(torch.rand((), generator=g)))
                m.bias.copy_(0.1 * torch.randn(m.bias.shape, generator=g))
            for m in [gen.rgb4, *gen.rgbs]:
                m.bias.copy_(0.1 * torch.randn(m.bias.shape, generator=g))
        gen = gen.to(DEV).eval()
        for p in gen.parameters():
            p.requires_grad_(False)
        _GENERATOR.append(gen)
    return _GENERATOR[0]


def _layer_of(case):
    """(layer, input side, input channels, output channels) of the generator's style layer with this output side."""
    gen = _generator()
    i = int(math.log2(case["res"])) - 3
    layer = gen.ups[i] if case["up"] else gen.convs[i]
    cout, cin = layer.conv.weight.shape[:2]
    return layer, case["res"] // 2 if case["up"] else case["res"], cin, cout


def _layer_inputs(case, seed):
    g = _rng(seed)
    _, side, cin, cout = _layer_of(case)
    b, r = case["batch"], case["res"]
    cl = torch.channels_last
    x = torch.randn(b, cin, side, side, generator=g, device=DEV).contiguous(memory_format=cl)
    w = torch.randn(b, 512, generator=g, device=DEV)
    noise = torch.randn(b, 1, r, r, generator=g, device=DEV)
    gy = torch.randn(b, cout, r, r, generator=g, device=DEV).contiguous(memory_format=cl)
    return x, w, noise, gy


def _latent_inputs(case, seed):
    g = _rng(seed)
    gen = _generator()
    b = case["batch"]
    with torch.no_grad():
        w = gen.map(torch.randn(b, gen.w_dim, generator=g, device=DEV))
    latent = (w[:, None].repeat(1, gen.num_ws, 1) + 0.05 * torch.randn(b, gen.num_ws, gen.w_dim, generator=g, device=DEV))
    noises = [torch.randn(b, 1, r, r, generator=g, device=DEV) for r in gen.noise_res]
    cam, lit = _views(case["views"], g)
    targets = torch.cat([_photos(_material(256, g), cam, lit, g) for _ in range(b)])
    return latent, noises, cam, lit, targets


def _render_inputs(case, seed):
    g = _rng(seed)
    tex = torch.cat([_material(case["res"], g) for _ in range(case["batch"])])
    cam, lit = _views(case["views"], g, case["coloc"])
    gout = None
    if case["grad"]:
        gout = torch.randn(case["batch"] * case["views"], 3, case["res"], case["res"], generator=g, device=DEV)
    return tex, cam, lit, gout


def _optim_inputs(case, seed):
    g = _rng(seed)
    sc = _capture(case["res"], case["views"], g)
    light = _light() * (0.8 + 0.4 * _uniform(g, 3)) if case["light"] else _light()
    # the reference's constant start, with the small random spread of a start from photos
    init = (sc.init + 0.05 * torch.randn(sc.init.shape, generator=g, device=DEV)).clamp(-1, 1).contiguous()
    return sc, light, init


def _descriptor_inputs(case, seed):
    g = _rng(seed)
    side = max(case["h"], case["w"])
    cam, lit = _views(case["views"], g)
    with torch.no_grad():
        r = gb.Microfacet(side, case["views"], SIZE_CM, [cam, lit, _light()], DEV)
        cut = lambda t: r.eval(t)[:, :, :case["h"], :case["w"]].contiguous()
        return cut(_material(side, g)), cut(_material(side, g))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "render":
        tex, cam, lit, gout = _render_inputs(case, seed)
        light = _light().requires_grad_(case["light"])
        r = gb.Microfacet(case["res"], case["views"], SIZE_CM, [cam, lit, light], DEV)
        return SimpleNamespace(case=case, r=r, tex=tex.requires_grad_(case["grad"]), light=light, gout=gout)
    if kind == "optim":
        sc, light, init = _optim_inputs(case, seed)
        r = gb.Microfacet(case["res"], case["views"], SIZE_CM, [sc.camera_pos, sc.light_pos, light], DEV)
        o = gb.SvbrdfOptim(DEV, r, loss=case["loss"], graph=True)
        o.load_targets(sc.targets)
        o.init_from_tex(init.clone())
        return SimpleNamespace(case=case, o=o, r=r, init=init, light=light)
    if kind == "batch":
        g = _rng(seed)
        mats = [_capture(res, v, g) for res, v in _batch_shapes(case, seed)]
        b = gb.BatchedOptim(mats, lr=0.01, loss=case["loss"], device=DEV, hist_len=case["iters"])
        b.capture(case["iters"])
        return SimpleNamespace(case=case, b=b)
    if kind == "descriptor":
        renders, targets = _descriptor_inputs(case, seed)
        d = gb.descriptor.VGGDescriptor(DEV, seed=0, mode=case["mode"])
        d.load(targets)
        return SimpleNamespace(case=case, d=d, renders=renders)
    if kind == "layer":
        x, w, noise, gy = _layer_inputs(case, seed)
        return SimpleNamespace(case=case, layer=_layer_of(case)[0], x=x.requires_grad_(True), w=w.requires_grad_(True),
                               noise=noise.requires_grad_(True), gy=gy)
    if kind == "latent":
        latent, noises, cam, lit, targets = _latent_inputs(case, seed)
        r = gb.Microfacet(256, case["views"], SIZE_CM, [cam, lit, _light()], DEV)
        o = gb.materialgan.MaterialGANOptim(DEV, r, _generator())
        o.load_targets(targets)
        o.init_from(latent=latent)
        o.noises = [n.requires_grad_(True) for n in noises]
        return SimpleNamespace(case=case, o=o, r=r)
    g = _rng(seed)
    r = gb.EnvmapRenderer([case["res"]] * 2, gb.envmap.synthetic_envmap(seed=seed), _material(case["tex"], g), device=DEV,
                          spp=case["spp"], seed=seed & 0xFFFF)
    return SimpleNamespace(case=case, r=r, angle=float(_uniform(g, 1) * 80 - 40))


# ------------------------------------------------------------------------------------------------ the calls
def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "render":
        out = s.r.eval(s.tex)
        if not case["grad"]:
            return [out]
        wrt = [s.tex, s.light] if case["light"] else [s.tex]
        return [out.detach(), *torch.autograd.grad(out, wrt, s.gout)]
    if kind == "optim":
        with torch.no_grad():
            s.o.textures.copy_(s.init)  # the fit starts from the same maps again
        s.r.update_light(s.light)
        s.o.optim(case["epochs"], 0.01, None, case["light"])
        out = [s.o.textures.detach(), s.o.exp_avg, s.o.exp_avg_sq, np.asarray(s.o.loss_image_list, dtype=np.float32)]
        return out + [s.r.light_pow.detach()] if case["light"] else out
    if kind == "batch":
        s.b.run(case["iters"])
        return [*s.b.tex, s.b.loss_hist]
    if kind == "descriptor":
        return list(s.d.loss_and_grad(s.renders))
    if kind == "layer":
        y = s.layer(s.x, s.w, s.noise)
        return [y.detach(), *torch.autograd.grad(y, (s.x, s.w, s.noise), s.gy)]
    if kind == "latent":
        tex = s.o.latent_to_textures()
        loss = s.o.compute_image_loss(s.r.eval(tex))
        return [tex.detach(), loss.detach(), *torch.autograd.grad(loss, [s.o.latent, *s.o.noises])]
    return [s.r.render_device(s.angle, 0.5)]


# ------------------------------------------------------------------------------------------------ their work
def _vgg(mode):
    """(name, cin, cout) and "pool" entries of the descriptor's stack, and its hooked layers."""
    d = gb.descriptor
    return (d.VGG19_TO_CONV4_2, d.REF_HOOKS) if mode == "reference" else (d.VGG19_TO_CONV4_1, d.HOOKS)


def _generator_flops(b):
    gen, n = _generator(), 0.0
    for layer, r in [(gen.conv4, 4), *((m, 8 << i) for i, m in enumerate(gen.ups)), *((m, 8 << i) for i, m in enumerate(gen.convs))]:
        n += 2.0 * layer.conv.weight.numel() * r * r
    for layer, r in [(gen.rgb4, 4), *((m, 8 << i) for i, m in enumerate(gen.rgbs))]:
        n += 2.0 * layer.conv.weight.numel() * r * r
    return b * n


def work(case):
    kind = case["kind"]
    if kind == "render":
        n, v = case["batch"] * case["res"] ** 2, case["views"]
        if not case["grad"]:
            return {"bytes": n * (36 + 12 * v), "flops": n * v * FLOPS_VIEW_FWD}
        # maps in, renders out; the gradient of the renders in, that of the maps out
        return {"bytes": n * (36 + 12 * v + 12 * v + 36), "flops": n * v * (FLOPS_VIEW_FWD + FLOPS_VIEW_STEP)}
    if kind in ("optim", "batch"):
        shapes = [(case["res"], case["views"])] if kind == "optim" else _batch_shapes(case, 0)
        k = case["epochs"] if kind == "optim" else case["iters"]
        # maps in and out, the targets in, both moments out (and in, where a run goes on from the last)
        state = 72 + (72 if kind == "optim" else 144)
        return {"bytes": sum(r * r * (state + 12 * v) for r, v in shapes),
                "flops": sum(r * r * v for r, v in shapes) * k * FLOPS_VIEW_STEP}
    if kind == "descriptor":
        layers, hooks = _vgg(case["mode"])
        h, w = (case["h"] // 2, case["w"] // 2) if case["mode"] == "config" else (case["h"], case["w"])
        v, flops, nbytes = case["views"], 0.0, 2 * 12 * case["views"] * case["h"] * case["w"]
        for item in layers:
            if item == "pool":
                h, w = h // 2, w // 2
                continue
            name, cin, cout = item
            flops += 2 * 2.0 * 9 * cin * cout * h * w * v
            nbytes += 2 * 2 * 9 * cin * cout
            if name in hooks:
                nbytes += 2 * v * h * w * cout  # the targets' features, in 16 bits
                if case["mode"] == "config":
                    flops += 2 * 2.0 * h * w * cout * cout * v
        return {"bytes": nbytes, "flops": flops}
    if kind == "layer":
        layer, side, cin, cout = _layer_of(case)
        b, r = case["batch"], case["res"]
        # forward: x in, y out; backward: x, y and y's gradient in, x's gradient out
        return {"bytes": 4.0 * b * (3 * cin * side * side + 3 * cout * r * r) + 8.0 * layer.conv.weight.numel(),
                "flops": 2 * 2.0 * b * layer.conv.weight.numel() * r * r}
    if kind == "latent":
        n = case["batch"] * 256 * 256
        return {"bytes": 8.0 * sum(p.numel() for p in _generator().parameters()) + n * (24 * case["views"] + 72),
                "flops": 2 * _generator_flops(case["batch"]) + n * case["views"] * (FLOPS_VIEW_FWD + FLOPS_VIEW_STEP)}
    # per camera sample: the ray, a bilinear fetch of 9 maps, two light samples with their BSDF values
    return {"bytes": 12 * case["res"] ** 2 + 36 * case["tex"] ** 2 + 12 * 64 * 128, "flops": 600.0 * case["res"] ** 2 * case["spp"]}


# ------------------------------------------------------------------------------------------------ in 64 bits
def _render64(tex, cam, lit, light):
    """The flash-lit GGX model in 64 bits: [B, 9, R, R] -> [B V, 3, R, R]."""
    res = tex.shape[-1]
    k = ((torch.arange(res, device=DEV, dtype=torch.float32) + 0.5) / res - 0.5) * SIZE_CM
    pos = torch.stack((k.expand(res, res), -k[:, None].expand(res, res), torch.zeros(res, res, device=DEV))).double()
    unit = lambda x: x / x.norm(dim=-3, keepdim=True)
    dot = lambda a, b: (a * b).sum(-3, keepdim=True)
    t = tex.double()
    lin = ((t + 1) / 2) ** 2.2
    dif, rgh, spe = lin[:, 0:3], lin[:, 5:6], lin[:, 6:9]
    nx, ny = t[:, 3:4].clamp(-1, 1), t[:, 4:5].clamp(-1, 1)
    nz = (1 - (nx * nx + ny * ny).clamp(0, 1 - EPS)).sqrt()
    n = unit(torch.cat((nx, ny, nz), 1))
    alpha = rgh * rgh
    out = []
    for b in range(t.shape[0]):
        for c, l in zip(cam.double(), lit.double()):
            tov, tol = c[:, None, None] - pos, l[:, None, None] - pos
            v, li = unit(tov), unit(tol)
            h = unit(v + li)
            nv, nl, nh, vh = (dot(x, y).clamp(min=0) for x, y in ((n[b], v), (n[b], li), (n[b], h), (v, h)))
            c2, a2 = nh * nh, alpha[b] * alpha[b]
            d = a2 / (math.pi * (c2 * a2 + (1 - c2)) ** 2 + EPS)
            f = spe[b] + (1 - spe[b]) * torch.exp2((-5.55473 * vh - 6.98316) * vh)
            kk = alpha[b] * 0.5 + EPS
            g = (nv / (nv * (1 - kk) + kk)) * (nl / (nl * (1 - kk) + kk))
            f1, f2 = dif[b] / math.pi * (1 - spe[b]), d * f * g / (4 * nv * nl + EPS)
            img = light.double()[:, None, None] * (f1 + f2) * nl / dot(tol, tol)
            out.append(img.clamp(EPS, 1) ** (1 / 2.2))
    return torch.stack(out)


def _fit64(sc, init, light, epochs, loss, learn_light):
    """The Adam loop in 64 bits, as plain torch runs it."""
    tex = init.double().clone().requires_grad_(True)
    light = light.double().clone().requires_grad_(learn_light)
    params = [tex, light] if learn_light else [tex]
    opt = torch.optim.Adam(params, lr=0.01, betas=(0.9, 0.999))
    squash = torch.log1p if loss == "log1p" else (lambda x: x)
    target, losses = squash(sc.targets.double()), []
    for _ in range(epochs):
        e = Fn.mse_loss(squash(_render64(tex.clamp(-1, 1), sc.camera_pos, sc.light_pos, light)), target)
        opt.zero_grad()
        e.backward()
        opt.step()
        losses.append(e.detach())
    st = opt.state[tex]
    return tex.detach(), st["exp_avg"], st["exp_avg_sq"], torch.stack(losses), light.detach()


def _layer64(layer, x, w, noise):
    """One style layer in 64 bits with the layer's weights: modulation, (up-sampling) convolution, demodulation, noise,
    bias, leaky ReLU."""
    m = layer.conv
    weight = m.weight.double() * m.scale
    style = w @ (m.affine.weight.double() * m.affine.scale).t() + m.affine.bias.double() * m.affine.lr_mul
    demod = torch.rsqrt(style ** 2 @ (weight ** 2).sum((2, 3)).t() + 1e-8)
    y = _conv64(x * style[:, :, None, None], weight, m.up) * demod[:, :, None, None]
    y = y + layer.noise_strength.double() * noise + layer.bias.double()[:, None, None]
    return Fn.leaky_relu(y, 0.2) * math.sqrt(2.0)


def _fir64(c):
    k = torch.tensor([1.0, 3.0, 3.0, 1.0], dtype=torch.float64, device=DEV) / 4
    return torch.outer(k, k).expand(c, 1, 4, 4)


def _conv64(x, weight, up):
    if not up:
        return Fn.conv2d(x, weight, padding=weight.shape[-1] // 2)
    # a stride-2 transposed convolution with the flipped kernel, then the [1, 3, 3, 1] filter
    y = Fn.conv_transpose2d(x, weight.flip(2, 3).transpose(0, 1), stride=2)
    return Fn.conv2d(Fn.pad(y, (1, 1, 1, 1)), _fir64(y.shape[1]), groups=y.shape[1])


def _image_up64(x):
    c = x.shape[1]
    z = torch.zeros(x.shape[0], c, 2 * x.shape[2], 2 * x.shape[3], dtype=torch.float64, device=DEV)
    z[:, :, ::2, ::2] = x
    return Fn.conv2d(Fn.pad(z, (2, 1, 2, 1)), _fir64(c), groups=c)


def _rgb64(layer, x, w):
    m = layer.conv
    style = w @ (m.affine.weight.double() * m.affine.scale).t() + m.affine.bias.double() * m.affine.lr_mul
    return Fn.conv2d(x * style[:, :, None, None], m.weight.double() * m.scale) + layer.bias.double()[:, None, None]


def _textures64(latent, noises):
    gen = _generator()
    x = gen.const.double().expand(latent.shape[0], -1, -1, -1)
    x = _layer64(gen.conv4, x, latent[:, 0], noises[0])
    img = _rgb64(gen.rgb4, x, latent[:, 1])
    for i, (up, conv, rgb) in enumerate(zip(gen.ups, gen.convs, gen.rgbs)):
        x = _layer64(up, x, latent[:, 1 + 2 * i], noises[1 + 2 * i])
        x = _layer64(conv, x, latent[:, 2 + 2 * i], noises[2 + 2 * i])
        img = _rgb64(rgb, x, latent[:, 3 + 2 * i]) + _image_up64(img)
    return torch.cat((img[:, 0:5].clamp(-1, 1), img[:, 5:6].clamp(-0.5, 0.5), img[:, 6:9].clamp(-1, 1)), 1)


def _vgg64(case, images, weights):
    """The hooked features of the stack in 64 bits."""
    layers, hooks = _vgg(case["mode"])
    x = images
    if case["mode"] == "config":
        x = Fn.avg_pool2d(x, 2)
    mean = torch.tensor(gb.descriptor.MEAN, dtype=torch.float64, device=DEV)[:, None, None]
    std = torch.tensor(gb.descriptor.STD, dtype=torch.float64, device=DEV)[:, None, None]
    x, out = (x - mean) / std, []
    for item in layers:
        if item == "pool":
            x = Fn.max_pool2d(x, 2) if case["mode"] == "config" else Fn.avg_pool2d(x, 2)
            continue
        w, b = weights[item[0]]
        x = torch.relu(Fn.conv2d(x, w.double().to(DEV), b.double().to(DEV), padding=1))
        if item[0] in hooks:
            out.append(x)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "render":
        tex, cam, lit, gout = _render_inputs(case, seed)
        if not case["grad"]:
            return [_render64(tex, cam, lit, _light())]
        outs, gtex, glight = [], [], torch.zeros(3, dtype=torch.float64, device=DEV)
        for b in range(case["batch"]):
            t, light = tex[b:b + 1].double().requires_grad_(True), _light().double().requires_grad_(True)
            for v in range(case["views"]):
                k = b * case["views"] + v
                o = _render64(t, cam[v:v + 1], lit[v:v + 1], light)
                o.backward(gout[k:k + 1].double())
                outs.append(o.detach())
            gtex.append(t.grad)
            glight += light.grad
        return [torch.cat(outs), torch.cat(gtex)] + ([glight] if case["light"] else [])
    if kind == "optim":
        if case["res"] ** 2 * case["views"] * case["epochs"] > 1.5e8:
            return None  # too long in 64 bits
        sc, light, init = _optim_inputs(case, seed)
        got = _fit64(sc, init, light, case["epochs"], case["loss"], case["light"])
        return list(got) if case["light"] else list(got[:4])
    if kind == "batch":
        shapes = _batch_shapes(case, seed)
        if sum(r * r * v for r, v in shapes) * case["iters"] > 1.5e8:
            return None  # too long in 64 bits
        g = _rng(seed)
        got = [_fit64(sc, sc.init, sc.light_pow, case["iters"], case["loss"], False)
               for sc in [_capture(r, v, g) for r, v in shapes]]
        return [x[0] for x in got] + [torch.stack([x[3] for x in got], 1)]
    if kind == "descriptor":
        renders, targets = _descriptor_inputs(case, seed)
        weights = gb.descriptor.VGGDescriptor(DEV, seed=0, mode=case["mode"]).bf16_weights()
        grad = case["mode"] == "reference"
        r = renders.double().requires_grad_(grad)
        with torch.no_grad():
            tf = _vgg64(case, targets.double(), weights)
        with torch.set_grad_enabled(grad):
            f = _vgg64(case, r, weights)
            w2 = 0.25 ** 2
            fl = sum(w2 * ((a - b) ** 2).sum() for a, b in zip(f, tf)) / sum(a.numel() for a in f)
        if grad:
            fl.backward()
            return [fl.detach(), None, r.grad]
        gram = lambda x: torch.bmm(x.flatten(2), x.flatten(2).transpose(1, 2)) / (x.shape[2] * x.shape[3])
        gl = sum(w2 * ((gram(a) - gram(b)) ** 2).sum() for a, b in zip(f, tf)) / sum(a.shape[0] * a.shape[1] ** 2 for a in f)
        # the gradient goes through max-pools, whose winners change with the features' rounding: 64 bits pick others
        return [fl, gl, None]
    if kind == "layer":
        x, w, noise, gy = _layer_inputs(case, seed)
        leaves = [t.double().requires_grad_(True) for t in (x, w, noise)]
        y = _layer64(_layer_of(case)[0], *leaves)
        return [y.detach(), *torch.autograd.grad(y, leaves, gy.double())]
    if kind == "latent":
        if case["batch"] > 4:
            return None  # too long in 64 bits
        latent, noises, cam, lit, targets = _latent_inputs(case, seed)
        leaves = [t.double().requires_grad_(True) for t in [latent, *noises]]
        tex = _textures64(leaves[0], leaves[1:])
        loss = Fn.mse_loss(_render64(tex, cam, lit, _light()), targets.double())
        return [tex.detach(), loss.detach(), *torch.autograd.grad(loss, leaves)]
    # every sample draws a texel of the environment: 64 bits draw another one where the choice is close
    return None
