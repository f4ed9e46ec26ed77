"""Timed cases of the framework's public entry points.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare(case, seed)`` makes a case's inputs, ``run(state)`` is one pass through the
public API, ``work(case)`` the bytes and operations a pass cannot do without, and
``exact(case, seed)`` the same outputs in float64 from plain torch operations.

What the cases stand for:

``render``      novel views and training steps of a stroke scene through
                ``field.render_strokes`` (sample positions given) or ``field.render_rays``
                (samples cast in the kernels): previews of a small scene, whole images of a
                large one, and forward + backward at the benchmark's sizes.
``field``       one training step of a model's ``StrokeField`` module (device-side stroke
                count, linear soft step, cone radii): the first strokes of a run, where
                launches and latency are all there is, and the full 500-stroke field.
``batch``       many uneven scenes per launch, ``train.BatchedField`` captured in a CUDA
                graph, as a program that fits several scenes at once runs it.
``operators``   the drop-in stroke and composition operators on dense [samples, strokes]
                tensors, for a model that keeps the reference's structure (colour fields
                and composition modes included).
``grid``        the multi-resolution hash-grid encoder, forward and table gradient.
``density``     one proposal or error network of a training step, hash decay included.
``sampling``    the proposal levels of a render call, two networks and three resamplings.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from neural3dstrokes_b200 import gridencoder, mlp, sampler, scenes, strokes, train
from neural3dstrokes_b200.field import render_rays, render_strokes
from neural3dstrokes_b200.strokefield import StrokeField

DEV = "cuda"
KIND_SETS = {
    "ellipsoid": ["ellipsoid"],
    "mixed": ["sphere", "cube", "roundcube", "tetrahedron", "octahedron", "capsule"],
    "curves": ["quadratic_bezier", "cubic_bezier"],
    "all": ["sphere", "cube", "roundcube", "tetrahedron", "octahedron", "capsule", "quadratic_bezier",
            "cubic_bezier"],
}


def listed():
    return [
        # a preview of a small scene while it is edited: 64 ellipsoids, no gradient
        dict(name="preview_ellipsoids", op="render", kinds="ellipsoid", strokes=64, rays=4096, samples=64, grad=False,
             cast=False),
        # the first steps of a run: 10 strokes of 500 placed, a ragged batch of rays
        dict(name="first_strokes", op="field", shape="sphere", active=10, strokes=500, rays=1003, samples=32),
        # a training step of the reference model's stroke level: 2^14 rays, 32 samples
        dict(name="train_field", op="field", shape="ellipsoid", active=500, strokes=500, rays=16384, samples=32),
        # forward + backward with position gradients, 500 mixed primitives
        dict(name="mixed_primitives", op="render", kinds="mixed", strokes=500, rays=65536, samples=128, grad=True,
             cast=False),
        # Bezier tubes, samples cast in the kernels, an odd number of rays
        dict(name="bezier_tubes", op="render", kinds="curves", strokes=2000, rays=16411, samples=64, grad=True,
             cast=True),
        # 16 uneven scenes in one graph, forward + backward
        dict(name="scene_batch", op="batch", kinds="mixed", scenes=16, max_strokes=2000, max_rays=65536, samples=64,
             size_seed=3),
        # a large view of a finished scene: primitives and curves, no gradient
        dict(name="full_view", op="render", kinds="all", strokes=2000, rays=131072, samples=96, grad=False, cast=True),
        # the drop-in operators at a model's chunk of samples, forward + backward
        dict(name="operators_cubes", op="operators", shape="cube", color="constant_rgb", compose="over", rays=1024,
             samples=64, strokes=256, laplace=True, grad_x=False),
        # a colour field and a soft composition, ragged strokes, position gradients
        dict(name="operators_sh3", op="operators", shape="capsule", color="constant_sh3",
             compose="softmax_density_weighted", rays=311, samples=64, strokes=131, laplace=False, grad_x=True),
        # the encoder's defaults on 2^20 ray-ordered points, one ray ragged
        dict(name="hash_grid", op="grid", levels=10, channels=4, resolution=8192, log2_rows=21, rays=16385, samples=64),
        # the second proposal network's share of a training step
        dict(name="density_network", op="density", resolution=2048, channels=1, log2_rows=21, rays=16384, samples=64),
        # the proposal levels of a render call
        dict(name="ray_sampling", op="sampling", rays=16384, prop_samples=64, samples=32),
    ]


def draw(rng):
    def lu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["render", "render", "render", "field", "batch", "operators", "operators", "grid", "density",
                     "sampling"])
    if op == "render":
        grad = rng.random() < 0.6
        c = dict(op=op, kinds=rng.choice(list(KIND_SETS)), strokes=lu(16, 2000), rays=lu(256, 131072),
                 samples=rng.randint(16, 128), grad=grad, cast=rng.random() < 0.5)
        cap = 2e9 if c["kinds"] in ("curves", "all") else (4e9 if grad else 1e10)
        while c["strokes"] * c["rays"] * c["samples"] > cap:
            c["rays"] = c["rays"] * 2 // 3
        return c
    if op == "field":
        n = lu(32, 1000)
        return dict(op=op, shape=rng.choice(["sphere", "ellipsoid", "cube", "roundcube", "capsule", "octahedron"]),
                    active=rng.randint(max(1, n // 10), n), strokes=n, rays=lu(256, 16384), samples=rng.randint(16, 64))
    if op == "batch":
        return dict(op=op, kinds=rng.choice(["ellipsoid", "mixed"]), scenes=rng.randint(2, 16),
                    max_strokes=lu(200, 2000), max_rays=lu(4096, 32768), samples=rng.randint(24, 80),
                    size_seed=rng.randrange(1 << 20))
    if op == "operators":
        return dict(op=op, shape=rng.choice(["sphere", "ellipsoid", "cube", "roundcube", "capsule", "tetrahedron"]),
                    color=rng.choice(["constant_rgb", "constant_rgb", "constant_sh2", "constant_sh3"]),
                    compose=rng.choice(["over", "over", "softmax", "softmax_density_weighted"]), rays=lu(32, 1024),
                    samples=rng.randint(16, 64), strokes=rng.randint(8, 256), laplace=rng.random() < 0.5,
                    grad_x=rng.random() < 0.5)
    if op == "grid":
        return dict(op=op, levels=rng.randint(4, 10), channels=rng.choice([1, 2, 4]), resolution=lu(256, 8192),
                    log2_rows=rng.randint(17, 21), rays=lu(512, 16384), samples=rng.randint(32, 64))
    if op == "density":
        ch = rng.choice([1, 1, 2])
        return dict(op=op, resolution=rng.choice([256, 512, 1024, 2048]) if ch == 1 else 256, channels=ch,
                    log2_rows=rng.randint(18, 21), rays=lu(512, 16384), samples=rng.randint(32, 64))
    return dict(op=op, rays=lu(512, 16384), prop_samples=rng.randint(24, 64), samples=rng.randint(16, 64))


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(g, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=g, device=DEV) * (hi - lo) + lo


def _normal(g, shape):
    return torch.randn(shape, generator=g, device=DEV)


def _log_uniform(g, shape, lo, hi):
    return torch.exp(_uniform(g, shape, math.log(lo), math.log(hi)))


def _kinds(pool, n, seed):
    pick = np.random.RandomState(int(seed) % (1 << 31)).randint(0, len(pool), n)
    return [pool[int(i)] for i in pick]


def _stroke_rows(kinds, g):
    """[S, 16] parameter rows in the framework's layouts, zero-padded."""
    n = len(kinds)
    centre, euler = _uniform(g, (n, 3), -1, 1), _uniform(g, (n, 3), -math.pi, math.pi)
    s1, s3 = _log_uniform(g, (n, 1), 0.05, 0.3), _log_uniform(g, (n, 3), 0.05, 0.3)
    rnd, half = _uniform(g, (n, 1), 0, 0.3), _log_uniform(g, (n, 1), 0.05, 0.3)
    tube = _uniform(g, (n, 1), 0.02, 0.1)
    ctrl = (centre[:, None] + _normal(g, (n, 4, 3)) * 0.15).reshape(n, 12)
    radii = _uniform(g, (n, 2), 0.01, 0.06)
    rows = {
        "sphere": [s1, centre], "ellipsoid": [s3, euler, centre], "cube": [s1, euler, centre],
        "octahedron": [s1, euler, centre], "tetrahedron": [s1, euler, centre], "roundcube": [rnd, s1, euler, centre],
        "capsule": [(half / tube).clamp_min(0.25), tube, euler, centre],
        "quadratic_bezier": [ctrl[:, :9], radii], "cubic_bezier": [ctrl, radii],
    }
    out = torch.zeros(n, 16, device=DEV)
    for k in sorted(set(kinds)):
        at = torch.tensor([i for i, q in enumerate(kinds) if q == k], device=DEV)
        row = torch.cat(rows[k], 1)
        out[at, :row.shape[1]] = row[at]
    return out


def _rays(n, samples, g, base_radius=None):
    """Rays from a sphere of radius 4 towards the scene with up to 0.5 rad of jitter and
    stratified fence posts in [2, 6]; sample radii 1, or those of cones."""
    u = F.normalize(_normal(g, (n, 3)), dim=-1)
    w = _normal(g, (n, 3))
    w = F.normalize(w + u * (w * -u).sum(-1, keepdim=True), dim=-1)
    th = _uniform(g, (n, 1), 0, 0.5)
    o, d = 4 * u, -u * torch.cos(th) + w * torch.sin(th)
    jit = _uniform(g, (n, samples + 1), -0.4, 0.4)
    jit[:, 0] = 0
    jit[:, -1] = 0
    td = 2 + (torch.arange(samples + 1, device=DEV) + jit) * (4.0 / samples)
    t = (td[:, :-1] + td[:, 1:]) / 2
    x = d[:, None] * t[..., None] + o[:, None]
    radii = _uniform(g, (n,), 0.5, 1.5) * base_radius if base_radius else torch.ones(n, device=DEV)
    radius = radii[:, None] * t if base_radius else torch.ones_like(t)
    return dict(o=o, d=d, radii=radii, td=td, x=x, radius=radius)


def _batch_sizes(case):
    r = np.random.RandomState(case["size_seed"])
    lo_s, lo_r = max(8, case["max_strokes"] // 40), max(64, case["max_rays"] // 16)
    s = np.exp(r.uniform(math.log(lo_s), math.log(case["max_strokes"]), case["scenes"]))
    n = np.exp(r.uniform(math.log(lo_r), math.log(case["max_rays"]), case["scenes"]))
    return [int(round(v)) for v in s], [int(round(v)) for v in n]


def _ray_points(n, samples, g):
    """Ray-ordered points of [-1, 1]^3 (rays through the box, clipped to it)."""
    r = _rays(n, samples, g)
    return (r["x"] / 2).clamp(-1, 1).reshape(-1, 3).contiguous()


def _network(resolution, channels, log2_rows, g):
    if channels == 1:
        net = mlp.PropMLP(grid_disired_resolution=resolution, grid_log2_hashmap_size=log2_rows)
    else:
        net = mlp.ErrorMLP(grid_disired_resolution=resolution, grid_log2_hashmap_size=log2_rows, disable_rgb=True)
    net = net.to(DEV)
    with torch.no_grad():
        for name, p in sorted(net.named_parameters()):
            p.copy_(_normal(g, p.shape) * 0.1 if "embeddings" in name else _uniform(g, p.shape, -0.4, 0.4))
    return net


def _net_params(net):
    return [net.encoder.embeddings, net.density_layer[0].weight, net.density_layer[0].bias,
            net.density_layer[2].weight, net.density_layer[2].bias]


def _render_weights(s, R, N, laplace):
    """Rendering weights [R, N] of the over-composited strokes, and interval length times
    transmittance (the size of a density's gradient)."""
    delta = torch.full((len(s["kinds"]),), s["delta"], device=DEV)
    white = torch.ones(len(s["kinds"]), 3, device=DEV)
    step = max(1, 4_000_000 // (N * len(s["kinds"])))
    dens = torch.cat([_over(*_alphas(s["kinds"], s["rays"]["x"][i:i + step].reshape(-1, 3),
                                     s["rays"]["radius"][i:i + step].reshape(-1), s["shape"], delta, laplace),
                            white, s["density"])[0] for i in range(0, R, step)]).reshape(R, N)
    dt = s["rays"]["td"][:, 1:] - s["rays"]["td"][:, :-1]
    tau = dens * dt
    trans = torch.exp(-(torch.cumsum(tau, 1) - tau))
    return -torch.expm1(-tau) * trans, dt * trans


def _inputs(case, seed):
    """Every tensor of a case, from the seed alone."""
    g, op = _gen(seed), case["op"]
    s = dict(case=case)
    if op == "render":
        kinds = _kinds(KIND_SETS[case["kinds"]], case["strokes"], seed)
        n, R = case["strokes"], case["rays"]
        s.update(kinds=kinds, shape=_stroke_rows(kinds, g), color=_uniform(g, (n, 3)),
                 density=_uniform(g, (n,), 5, 15), rays=_rays(R, case["samples"], g, 0.25 if case["cast"] else None),
                 g_rgb=_normal(g, (R, 3)), g_acc=_normal(g, (R,)), delta=0.02, bg=1.0)
    elif op == "field":
        n, R = case["strokes"], case["rays"]
        kinds = [case["shape"]] * n
        s.update(kinds=kinds, shape=_stroke_rows(kinds, g)[:, :scenes.N_PARAMS[case["shape"]]].contiguous(),
                 color=_uniform(g, (n, 3)), density=_uniform(g, (n,), 0.5, 1.5),
                 rays=_rays(R, case["samples"], g, base_radius=0.001), g_rgb=_normal(g, (R, 3)),
                 g_acc=_normal(g, (R,)), bg=_uniform(g, (R, 3)))
    elif op == "batch":
        ns, nr = _batch_sizes(case)
        s["scenes"] = []
        for i, (n, R) in enumerate(zip(ns, nr)):
            kinds = _kinds(KIND_SETS[case["kinds"]], n, seed * 64 + i)
            s["scenes"].append(dict(kinds=kinds, shape=_stroke_rows(kinds, g), color=_uniform(g, (n, 3)),
                                    density=_uniform(g, (n,), 5, 15), rays=_rays(R, case["samples"], g),
                                    g_rgb=_normal(g, (R, 3)), g_acc=_normal(g, (R,)), delta=0.02, bg=1.0))
    elif op == "operators":
        n, R, N = case["strokes"], case["rays"], case["samples"]
        kinds = [case["shape"]] * n
        n_col = {"constant_rgb": 3, "constant_sh2": 12, "constant_sh3": 27}[case["color"]]
        col = _uniform(g, (n, 3)) if n_col == 3 else _normal(g, (n, n_col))
        s.update(kinds=kinds, shape=_stroke_rows(kinds, g)[:, :scenes.N_PARAMS[case["shape"]]].contiguous(), color=col,
                 density=_uniform(g, (n,), 0.5, 1.5), rays=_rays(R, N, g), delta=0.05 if case["laplace"] else 0.1)
        # upstream gradients as a rendering loss gives them: scaled by the samples' weights
        with torch.no_grad():
            w, reach = _render_weights(s, R, N, case["laplace"])
        s.update(g_dens=_normal(g, (R, N)) * reach, g_col=_normal(g, (R, N, 3)) * w[..., None])
    elif op == "grid":
        s["points"] = _ray_points(case["rays"], case["samples"], g)
        s["g_out"] = _normal(g, (s["points"].shape[0], case["levels"] * case["channels"]))
        s["encoder"] = gridencoder.GridEncoder(input_dim=3, num_levels=case["levels"], level_dim=case["channels"],
                                               base_resolution=16, desired_resolution=case["resolution"],
                                               log2_hashmap_size=case["log2_rows"]).to(DEV)
        with torch.no_grad():
            s["encoder"].embeddings.copy_(_normal(g, s["encoder"].embeddings.shape) * 0.1)
    elif op == "density":
        s["net"] = _network(case["resolution"], case["channels"], case["log2_rows"], g)
        s["points"] = (_rays(case["rays"], case["samples"], g)["x"]).contiguous()
        s["g_dens"] = _normal(g, s["points"].shape[:-1])
        L, C = s["net"].encoder.num_levels, case["channels"]
        s["g_hash"] = _uniform(g, (L, C))
    else:
        s["nets"] = [_network(512, 1, 21, g).eval(), _network(2048, 1, 21, g).eval()]
        r = _rays(case["rays"], 2, g, base_radius=0.001)
        s.update(o=r["o"], d=r["d"], radii=r["radii"], near=torch.full((case["rays"],), 2.0, device=DEV),
                 far=torch.full((case["rays"],), 6.0, device=DEV))
    return s


def prepare(case, seed):
    s, op = _inputs(case, seed), case["op"]
    if op == "render":
        s["ids"] = torch.tensor([scenes.SDF_ID[k] for k in s["kinds"]], dtype=torch.int32, device=DEV)
        if case["grad"]:
            for k in ("shape", "color", "density"):
                s[k].requires_grad_(True)
            if not case["cast"]:
                s["rays"]["x"].requires_grad_(True)
    elif op == "field":
        m = StrokeField(case["shape"], max_num_strokes=case["strokes"], max_opt_strokes=case["strokes"]).to(DEV)
        with torch.no_grad():
            m.shape_params.copy_(s["shape"])
            m.color_params.copy_(s["color"])
            m.density_params.copy_(s["density"])
            m.stroke_step.fill_(case["active"])
        s["module"] = m.train()
    elif op == "batch":
        sc, rs = [], []
        for q in s["scenes"]:
            ids = torch.tensor([scenes.SDF_ID[k] for k in q["kinds"]], dtype=torch.int32, device=DEV)
            r = q["rays"]
            sc.append(scenes.Scene(q["kinds"], ids, q["shape"], q["color"], q["density"]))
            rs.append(scenes.RaySet(r["o"], r["d"], r["td"], r["x"], r["radius"]))
        f = train.BatchedField(sc, rs, sdf_delta=s["scenes"][0]["delta"], bg=s["scenes"][0]["bg"])
        f.g_rgb.copy_(torch.cat([q["g_rgb"] for q in s["scenes"]]))
        f.g_acc.copy_(torch.cat([q["g_acc"] for q in s["scenes"]]))
        s = dict(case=case, batched=f, graph=train.capture(f.step))
    elif op == "operators":
        s["fn"] = strokes.get_stroke(case["shape"], case["color"], "recon")[0]
        for k in ("shape", "color", "density"):
            s[k].requires_grad_(True)
        if case["grad_x"]:
            s["rays"]["x"].requires_grad_(True)
    return s


# ------------------------------------------------------------------ one pass

def _run_render(s):
    c, r = s["case"], s["rays"]
    if c["cast"]:
        out = render_rays(r["o"], r["d"], r["radii"], r["td"], s["shape"], s["ids"], s["color"], s["density"],
                          s["delta"], bg=s["bg"])
    else:
        out = render_strokes(r["x"], r["radius"], r["td"], r["d"], s["shape"], s["ids"], s["color"], s["density"],
                             s["delta"], bg=s["bg"])
    res = dict(rgb=out[0], acc=out[1], depth=out[2])
    if c["grad"]:
        leaves = [s["shape"], s["color"], s["density"]] + ([] if c["cast"] else [r["x"]])
        g = torch.autograd.grad(out[:2], leaves, (s["g_rgb"], s["g_acc"]))
        res.update(zip(("grad_shape", "grad_color", "grad_density", "grad_x"), g))
    return res


def _run_field(s):
    m, r = s["module"], s["rays"]
    out = m.render(r["x"], r["radius"], r["td"], r["d"], bg=s["bg"])
    g = torch.autograd.grad(out[:2], [m.shape_params, m.color_params, m.density_params], (s["g_rgb"], s["g_acc"]))
    return dict(rgb=out[0], acc=out[1], depth=out[2], grad_shape=g[0], grad_color=g[1], grad_density=g[2])


def _run_operators(s):
    c, r = s["case"], s["rays"]
    alpha, color, _, _ = s["fn"](r["x"], r["radius"], r["d"], s["shape"], s["color"], s["delta"], c["laplace"], True)
    dens, col = strokes.compose_strokes(alpha, color, s["density"], c["compose"])
    leaves = [s["shape"], s["color"], s["density"]] + ([r["x"]] if c["grad_x"] else [])
    g = torch.autograd.grad((dens, col), leaves, (s["g_dens"], s["g_col"]))
    res = dict(alpha=alpha, density=dens, color=col)
    if c["color"] != "constant_rgb":
        res["stroke_color"] = color
    res.update(zip(("grad_shape", "grad_color", "grad_density", "grad_x"), g))
    return res


def run(s):
    op = s["case"]["op"]
    if op == "render":
        return _run_render(s)
    if op == "field":
        return _run_field(s)
    if op == "batch":
        s["graph"].replay()
        f = s["batched"]
        return dict(rgb=f.rgb, acc=f.acc, depth=f.depth, grad_x=f.grad_x, grad_shape=f.grad_shape,
                    grad_color=f.grad_color, grad_density=f.grad_density, grad_delta=f.grad_delta)
    if op == "operators":
        return _run_operators(s)
    if op == "grid":
        out = s["encoder"](s["points"])
        return dict(out=out, grad_table=torch.autograd.grad(out, s["encoder"].embeddings, s["g_out"])[0])
    if op == "density":
        out = s["net"](s["points"], None)
        g = torch.autograd.grad((out["density"], out["hash_levelwise_mean"]), _net_params(s["net"]),
                                (s["g_dens"], s["g_hash"]))
        return dict(density=out["density"], hash_mean=out["hash_levelwise_mean"], grads=list(g))
    with torch.no_grad():
        r = sampler.sample_rays(s["o"], s["d"], s["radii"], s["near"], s["far"], s["nets"],
                                num_prop_samples=s["case"]["prop_samples"], num_nerf_samples=s["case"]["samples"])
    return dict(sdist=r.sdist, tdist=r.tdist, density=[v["density"] for v in r.levels],
                weights=[v["weights"] for v in r.levels])


# ------------------------------------------------------------------ work

# Share of the nominal (sample, stroke) pairs within a stroke's reach in these scenes
# (strokes of 0.05 - 0.3 in a box of 2): the others have no effect on any output.
REACH = 0.027
PAIR_FLOPS = {"ellipsoid": 52, "mixed": 43, "curves": 148, "all": 70}


def _render_work(case, rays, n_strokes, kinds, grad, grad_x, cast, row):
    P = rays * case["samples"]
    b = rays * (case["samples"] + 1) * 4 + rays * (28 if cast else 12) + (0 if cast else P * 16) + rays * 20
    b += n_strokes * (row + 5) * 4
    pairs = P * n_strokes * REACH
    if not grad:
        return b, pairs * PAIR_FLOPS[kinds]
    return b + rays * 16 + n_strokes * (row + 5) * 4 + (P * 12 if grad_x else 0), pairs * PAIR_FLOPS[kinds] * 3.5


def work(case):
    op = case["op"]
    if op == "render":
        b, f = _render_work(case, case["rays"], case["strokes"], case["kinds"], case["grad"],
                            case["grad"] and not case["cast"], case["cast"], 16)
    elif op == "field":
        b, f = _render_work(case, case["rays"], case["active"], "ellipsoid", True, False, False,
                            scenes.N_PARAMS[case["shape"]])
    elif op == "batch":
        b = f = 0
        for n, R in zip(*_batch_sizes(case)):
            q = _render_work(case, R, n, case["kinds"], True, True, False, 16)
            b, f = b + q[0], f + q[1]
    elif op == "operators":
        # the operators' interface is the dense [samples, strokes] tensors: alpha and
        # colour written and read forward, both gradients written and read backward
        P, S = case["rays"] * case["samples"], case["strokes"]
        b = P * S * 16 * 4 + P * 16 * 3
        f = P * S * 50 * 3.5
    elif op == "grid":
        P, C, L = case["rays"] * case["samples"], case["channels"], case["levels"]
        rows = _grid_rows(L, case["resolution"], case["log2_rows"])
        b = P * 12 * 2 + P * L * C * 4 * 2 + rows * C * 4 * 2
        f = P * L * C * 8 * 2 * 2
    elif op == "density":
        P, C = case["rays"] * case["samples"], case["channels"]
        L = int(math.log(case["resolution"] / 16) / math.log(2)) + 1
        rows = _grid_rows(L, case["resolution"], case["log2_rows"])
        b = P * (12 * 2 + 4 * 2 + 12) + rows * C * 4 * 3
        f = P * (L * C * 64 * 2 + 128) * 3 + P * L * C * 8 * 4
    else:
        P = case["rays"] * case["prop_samples"]
        b = case["rays"] * 40 + 2 * P * 8 + case["rays"] * (case["samples"] + 1) * 8
        f = 2 * P * 8 * 64 * 2
    return dict(bytes=b, flops=f)


def _grid_rows(L, resolution, log2_rows):
    s = 2 ** (math.log2(resolution / 16) / (L - 1))
    return sum(min(2 ** log2_rows, (math.ceil(16 * s ** i) + 1) ** 3) for i in range(L))


# ------------------------------------------------------------------ float64

def _dot(a, b):
    return (a * b).sum(-1)


def _clamp01(t):
    return t.clamp(0, 1)


def _rotation(e):
    (sx, sy, sz), (cx, cy, cz) = torch.sin(e).unbind(-1), torch.cos(e).unbind(-1)
    rows = [cy * cz, sx * sy * cz - cx * sz, sx * sz + cx * sy * cz, cy * sz, cx * cz + sx * sy * sz,
            cx * sy * sz - sx * cz, -sy, sx * cy, cx * cy]
    return torch.stack(rows, -1).reshape(-1, 3, 3)


def _sdf(kind, x, prm):
    """(SDF, soft-step width factor) of points x [P, 3] and one kind's rows [n, d]."""
    if kind in ("quadratic_bezier", "cubic_bezier"):
        return (_quadratic if kind == "quadratic_bezier" else _cubic)(x, prm), torch.ones_like(prm[:, 0])
    nb = {"roundcube": 1, "capsule": 1}.get(kind, 0)
    s = prm[:, nb:nb + 3] if kind == "ellipsoid" else prm[:, nb:nb + 1].expand(-1, 3)
    k = nb + (3 if kind == "ellipsoid" else 1)
    e = None if kind == "sphere" else prm[:, k:k + 3]
    k += 0 if e is None else 3
    t = prm[:, k:k + 3]
    m = torch.eye(3, device=x.device, dtype=x.dtype).expand(len(t), 3, 3) if e is None else _rotation(e)
    p = [(x @ m[:, :, i].T - _dot(t, m[:, :, i])) / s[:, i] for i in range(3)]
    n2 = p[0] * p[0] + p[1] * p[1] + p[2] * p[2]
    width = s[:, 0]
    if kind in ("sphere", "ellipsoid"):
        if kind == "ellipsoid":
            width = torch.sqrt(sum((p[i] * s[:, i]) ** 2 for i in range(3))) / torch.sqrt(n2)
        return torch.sqrt(n2 + 1e-8) - 1, width
    if kind in ("cube", "roundcube"):
        q = [v.abs() - 1 for v in p]
        out = sum(v.clamp_min(0) ** 2 for v in q)
        inner = torch.maximum(q[0], torch.maximum(q[1], q[2])).clamp_max(0)
        if kind == "roundcube":
            return torch.sqrt(out + 1e-8) + inner - prm[:, 0], width
        pos = out > 0
        return torch.where(pos, torch.sqrt(torch.where(pos, out, 1.0)), 0.0) + inner, width
    if kind == "capsule":
        h = prm[:, 0]
        y = p[1] - torch.minimum(torch.maximum(p[1], -h), h)
        return torch.sqrt(p[0] * p[0] + y * y + p[2] * p[2] + 1e-8) - 1, width
    kf = 0.57735027
    if kind == "octahedron":
        return (p[0].abs() + p[1].abs() + p[2].abs() - 1) * kf, width
    return (torch.maximum((p[0] + p[1]).abs() - p[2], (p[0] - p[1]).abs() + p[2]) - 1) * kf, width


def _quadratic(x, prm):
    """Distance to a quadratic Bezier tube by the closed-form stationary parameter, with
    the definition's regularisers."""
    A, B, C = prm[:, 0:3], prm[:, 3:6], prm[:, 6:9]
    a, b = B - A, A - 2 * B + C
    d = [A[:, i] - x[:, i:i + 1] for i in range(3)]
    kk = 1 / _dot(b, b)
    kx = kk * _dot(a, b)
    db, da = sum(d[i] * b[:, i] for i in range(3)), sum(d[i] * a[:, i] for i in range(3))
    ky, kz = kk * (2 * _dot(a, a) + db) / 3, kk * da
    p = ky - kx * kx
    q = kx * (2 * kx * kx - 3 * ky) + kz
    h = q * q + 4 * p ** 3
    one = h >= 0

    def dist2(t):
        return sum((d[i] + (2 * a[:, i] + b[:, i] * t) * t) ** 2 for i in range(3))

    def cbrt(v):
        av = torch.where(v != 0, v.abs(), 1.0)
        return torch.where(v != 0, torch.sign(v) * av ** (1 / 3), 0.0)

    H = torch.sqrt(torch.where(one, h, 0.0) + 1e-8)
    t1 = _clamp01(cbrt((H - q) / 2) + cbrt(-(H + q) / 2) - kx)
    z = torch.sqrt(torch.where(one, 1.0, -p) + 1e-8)
    v = torch.acos(torch.where(one, 0.0, q / (p * z * 2 + 1e-8)).clamp(-1 + 1e-15, 1 - 1e-15)) / 3
    m, n = torch.cos(v), torch.sin(v) * 1.732050808
    ta, tb = _clamp01((m + n) * z - kx), _clamp01((-n - m) * z - kx)
    e1, ea, eb = dist2(t1), dist2(ta), dist2(tb)
    t = torch.where(one, t1, torch.where(eb < ea, tb, ta))
    e = torch.where(one, e1, torch.minimum(ea, eb))
    return torch.sqrt(e + 1e-8) - (prm[:, 9] + t * (prm[:, 10] - prm[:, 9]))


def _cubic(x, prm):
    """Distance to a cubic Bezier tube at the parameter of the closest point of its
    10-piece polyline."""
    P = [prm[:, 3 * k:3 * k + 3] for k in range(4)]

    def point(t):
        u = 1 - t
        w = (u * u * u, 3 * u * u * t, 3 * u * t * t, t * t * t)
        return [sum(w[k] * P[k][:, i] for k in range(4)) for i in range(3)]

    best = tmin = None
    s0 = point(0.0)
    for i in range(1, 11):
        s1 = point(i * 0.1)
        ab = [s1[j] - s0[j] for j in range(3)]
        l2 = sum(v * v for v in ab)
        w = [x[:, j:j + 1] - s0[j] for j in range(3)]
        tt = _clamp01(sum(w[j] * ab[j] for j in range(3)) / l2)
        with torch.no_grad():
            d2 = sum((w[j] - ab[j] * tt) ** 2 for j in range(3))
        t = (i - 1) * 0.1 * (1 - tt) + i * 0.1 * tt
        if best is None:
            best, tmin = d2, t
        else:
            near = d2 < best
            best, tmin = torch.where(near, d2, best), torch.where(near, t, tmin)
        s0 = s1
    c = point(tmin)
    dist = torch.sqrt(sum((c[j] - x[:, j:j + 1]) ** 2 for j in range(3)))
    return dist - (prm[:, 12] + tmin * (prm[:, 13] - prm[:, 12]))


def _alphas(kinds, x, radius, shape, delta, laplace):
    """alpha and log(1 - alpha) [P, S] in stroke order."""
    parts, order = [], []
    for k in sorted(set(kinds)):
        at = [i for i, q in enumerate(kinds) if q == k]
        sdf, width = _sdf(k, x, shape[at])
        parts.append(-sdf * (2.0 if laplace else 0.5) * width / (delta[at] * radius[:, None]))
        order += at
    m = torch.cat(parts, 1)
    if order != sorted(order):
        m = m[:, torch.argsort(torch.tensor(order, device=x.device))]
    if not laplace:
        a = (m + 0.5).clamp(0, 0.9999)
        return a, torch.log1p(-a)
    e = 0.5 * torch.exp(-m.abs())
    return torch.where(m <= 0, e, 1 - e), torch.where(m <= 0, torch.log1p(-e), -math.log(2.0) - m)


ONE_EPS = float(np.float32(1.0) + np.float32(1e-6))


def _over(a, l1m, color, density):
    total = l1m.sum(1)
    w = a * torch.exp(total[:, None] - torch.cumsum(l1m, 1))
    col = w @ color if color.dim() == 2 else torch.einsum("ps,psc->pc", w, color)
    return w @ density, (col / (ONE_EPS - torch.exp(total))[:, None]).clamp(0, 1)


def _volume(sigma, col, td, dirs, bg):
    tau = sigma * (td[:, 1:] - td[:, :-1]) * dirs.norm(dim=-1, keepdim=True)
    alpha = -torch.expm1(-tau)
    trans = torch.exp(-torch.cat([torch.zeros_like(tau[:, :1]), torch.cumsum(tau[:, :-1], 1)], 1))
    w = alpha * trans
    acc = w.sum(1)
    rgb = (w[..., None] * col).sum(1) + (1 - acc).clamp_min(0)[:, None] * bg
    depth = (w * (td[:, 1:] + td[:, :-1]) / 2).sum(1) / acc.clamp_min(float(np.float32(1.1920929e-07)))
    return rgb, acc, torch.minimum(torch.maximum(depth, td[:, 0]), td[:, -1])


def _exact_render(s, laplace, grad, grad_x, chunk):
    """rgb, acc, depth and the gradients of one scene in float64."""
    r = {k: v.detach().double() for k, v in s["rays"].items()}
    leaves = [s[k].detach().double().requires_grad_(grad) for k in ("shape", "color", "density")]
    shape, color, density = leaves
    delta = s["delta"]
    delta = delta.double() if torch.is_tensor(delta) else torch.full((len(density),), float(np.float32(delta)),
                                                                     device=DEV, dtype=torch.float64)
    delta = delta.requires_grad_(grad)
    leaves.append(delta)
    R, N = r["radius"].shape
    if s.get("cast"):  # cast_rays: t, then the position, in float32 as the inputs are
        t32 = (s["rays"]["td"][:, :-1] + s["rays"]["td"][:, 1:]) * 0.5
        r["x"] = (s["rays"]["d"][:, None] * t32[..., None] + s["rays"]["o"][:, None]).double()
        r["radius"] = (s["rays"]["radii"][:, None] * t32).double()
    step = max(1, chunk // (N * max(1, len(density))))
    outs, gx, sums = [], [], [torch.zeros_like(v) for v in leaves]
    for i in range(0, R, step):
        at = slice(i, min(R, i + step))
        with torch.set_grad_enabled(grad):
            x = r["x"][at].reshape(-1, 3).clone().requires_grad_(grad_x)
            a, l1m = _alphas(s["kinds"], x, r["radius"][at].reshape(-1), shape, delta, laplace)
            sg, col = _over(a, l1m, color, density)
            n = r["td"][at].shape[0]
            bg = s["bg"][at].double() if torch.is_tensor(s["bg"]) else s["bg"]
            o = _volume(sg.reshape(n, N), col.reshape(n, N, 3), r["td"][at], r["d"][at], bg)
            if grad:
                loss = (o[0] * s["g_rgb"][at]).sum() + (o[1] * s["g_acc"][at]).sum()
                got = torch.autograd.grad(loss, leaves + ([x] if grad_x else []))
                for acc, v in zip(sums, got):
                    acc += v
                if grad_x:
                    gx.append(got[-1].reshape(n, N, 3))
        outs.append([v.detach() for v in o])
    res = dict(zip(("rgb", "acc", "depth"), (torch.cat(v) for v in zip(*outs))))
    if grad:
        res.update(grad_shape=sums[0], grad_color=sums[1], grad_density=sums[2], grad_delta=sums[3])
        if grad_x:
            res["grad_x"] = torch.cat(gx)
    return res


def _exact_field(case, s):
    n = case["active"]
    frac = min(max(n / case["strokes"], 0.0), 1.0)
    delta = float(np.float32(7.0 * (1 - frac) + 1.0 * frac))
    q = dict(s, kinds=s["kinds"][:n], shape=s["shape"][:n], color=s["color"][:n],
             density=s["density"][:n].double() * 20.0, delta=delta)
    q["rays"] = dict(s["rays"], x=s["rays"]["x"] / 2.0)  # the module's box of size 4
    res = _exact_render(q, False, True, False, 6_000_000)
    res["grad_density"] = res["grad_density"] * 20.0
    del res["grad_delta"]
    for k in ("grad_shape", "grad_color", "grad_density"):
        full = torch.zeros((case["strokes"],) + tuple(res[k].shape[1:]), device=DEV, dtype=torch.float64)
        full[:n] = res[k]
        res[k] = full
    return res


def _sh(n, d):
    x, y, z = d.unbind(-1)
    c0, c1 = 0.5 / math.sqrt(math.pi), math.sqrt(3 / math.pi) / 2
    w = [torch.full_like(x, c0), -c1 * y, c1 * z, -c1 * x]
    if n == 9:
        c2, c20, c22 = math.sqrt(15 / math.pi) / 2, math.sqrt(5 / math.pi) / 4, math.sqrt(15 / math.pi) / 4
        w += [c2 * x * y, -c2 * y * z, c20 * (3 * z * z - 1), -c2 * x * z, c22 * (x * x - y * y)]
    return torch.stack(w, -1)


def _exact_operators(case, s):
    R, N, S = case["rays"], case["samples"], case["strokes"]
    leaves = [s[k].detach().double().requires_grad_(True) for k in ("shape", "color", "density")]
    shape, colorp, density = leaves
    delta = torch.full((S,), float(np.float32(s["delta"])), device=DEV, dtype=torch.float64)
    outs, gx, sums = [], [], [torch.zeros_like(v) for v in leaves]
    step = max(1, 4_000_000 // (N * S))
    for i in range(0, R, step):
        at = slice(i, min(R, i + step))
        x = s["rays"]["x"].detach()[at].double().reshape(-1, 3).requires_grad_(case["grad_x"])
        n = len(x) // N
        a, l1m = _alphas(s["kinds"], x, s["rays"]["radius"][at].double().reshape(-1), shape, delta, case["laplace"])
        if case["color"] == "constant_rgb":
            color = colorp
        else:
            nb = colorp.shape[1] // 3
            w = _sh(nb, s["rays"]["d"][at].double())
            color = torch.sigmoid(torch.einsum("rb,sbc->rsc", w, colorp.reshape(S, nb, 3)))
            color = color[:, None].expand(n, N, S, 3).reshape(n * N, S, 3)
        if case["compose"] == "over":
            dens, col = _over(a, l1m, color, density)
        else:
            key = a * density if case["compose"] == "softmax_density_weighted" else a
            w = torch.softmax(key / 0.05, 1)
            dens = (w * a * density).sum(1)
            col = w @ color if color.dim() == 2 else torch.einsum("ps,psc->pc", w, color)
        loss = (dens * s["g_dens"][at].reshape(-1)).sum() + (col * s["g_col"][at].reshape(-1, 3)).sum()
        got = torch.autograd.grad(loss, leaves + ([x] if case["grad_x"] else []))
        for acc, v in zip(sums, got):
            acc += v
        if case["grad_x"]:
            gx.append(got[-1].reshape(n, N, 3))
        out = [a.reshape(n, N, S), dens.reshape(n, N), col.reshape(n, N, 3)]
        if case["color"] != "constant_rgb":
            out.append(color.reshape(n, N, S, 3))
        outs.append([v.detach() for v in out])
    res = dict(zip(("alpha", "density", "color", "stroke_color"), (torch.cat(v) for v in zip(*outs))))
    res.update(grad_shape=sums[0], grad_color=sums[1], grad_density=sums[2])
    if case["grad_x"]:
        res["grad_x"] = torch.cat(gx)
    return res


def _grid_corners(u, enc):
    """Per level: (rows [P, 8], weights [P, 8]) of points u in [0, 1]^3; positions in the
    precision of u."""
    M32, primes = 0xFFFFFFFF, (1, 2654435761, 805459861)
    S = np.float32(np.log2(enc.per_level_scale))
    inside = ((u >= 0) & (u <= 1)).all(-1)
    for lv in range(enc.num_levels):
        lo, hi = int(enc.offsets[lv]), int(enc.offsets[lv + 1])
        scale = np.float32(float(np.float32(2.0 ** float(np.float32(lv) * S))) * enc.base_resolution - 1.0)
        res = int(math.ceil(float(scale))) + 1
        pos = (u.double() * float(scale) + 0.5).to(u.dtype).double()
        cell = torch.floor(pos)
        fr, cell = pos - cell, cell.long()
        rows, wts = [], []
        for corner in range(8):
            c = [cell[:, d] + ((corner >> d) & 1) for d in range(3)]
            w = 1.0
            for d in range(3):
                w = w * (fr[:, d] if (corner >> d) & 1 else 1 - fr[:, d])
            stride, index = 1, torch.zeros_like(c[0])
            for d in range(3):
                if stride > hi - lo:
                    break
                index = (index + c[d] * stride) & M32
                stride = (stride * (res + 1)) & M32
            if stride > hi - lo:
                index = c[0] ^ ((c[1] * primes[1]) & M32) ^ ((c[2] * primes[2]) & M32)
            rows.append(index % (hi - lo) + lo)
            wts.append(torch.where(inside, w, 0.0))
        yield torch.stack(rows, 1), torch.stack(wts, 1)


def _exact_features(u, enc, table):
    return torch.cat([(table[rows] * w[..., None]).sum(1) for rows, w in _grid_corners(u, enc)], -1)


def _exact_grid(s):
    enc = s["encoder"]
    u = (s["points"] + 1) / 2
    table = enc.embeddings.detach().double()
    C, grad = table.shape[1], torch.zeros_like(table)
    outs = []
    for lv, (rows, w) in enumerate(_grid_corners(u, enc)):
        outs.append((table[rows] * w[..., None]).sum(1))
        g = s["g_out"][:, lv * C:(lv + 1) * C].double()
        grad.index_add_(0, rows.reshape(-1), (w[..., None] * g[:, None]).reshape(-1, C))
    return dict(out=torch.cat(outs, -1), grad_table=grad)


def _contract(x):
    m = torch.sum(x ** 2, dim=-1, keepdim=True).clamp_min(torch.finfo(torch.float32).eps)
    return torch.where(m <= 1, x, ((2 * torch.sqrt(m) - 1) / m) * x) / 2.0


def _layers(feat, p):
    return F.softplus((torch.relu(feat @ p[1].T + p[2]) @ p[3].T + p[4])[..., 0] - 1.0, threshold=1e9)


def _exact_density(s):
    net = s["net"]
    u = (_contract(s["points"].reshape(-1, 3)) + 1) / 2
    p = [v.detach().double() for v in _net_params(net)]
    feat = _exact_features(u, net.encoder, p[0]).requires_grad_(True)
    leaves = [v.requires_grad_(True) for v in p[1:]]
    dens = _layers(feat, [p[0]] + leaves)
    got = torch.autograd.grad(dens, [feat] + leaves, s["g_dens"].double().reshape(-1))
    C, g_table = p[0].shape[1], torch.zeros_like(p[0])
    mean = torch.zeros(net.encoder.num_levels, C, device=DEV, dtype=torch.float64)
    for lv, (rows, w) in enumerate(_grid_corners(u, net.encoder)):
        g = got[0][:, lv * C:(lv + 1) * C]
        g_table.index_add_(0, rows.reshape(-1), (w[..., None] * g[:, None]).reshape(-1, C))
        lo, hi = int(net.encoder.offsets[lv]), int(net.encoder.offsets[lv + 1])
        mean[lv, 0] = (p[0][lo:hi, 0] ** 2).mean()
        g_table[lo:hi, 0] += s["g_hash"][lv, 0] * 2 * p[0][lo:hi, 0] / (hi - lo)
    return dict(density=dens.detach().reshape(s["points"].shape[:-1]), hash_mean=mean, grads=[g_table] + list(got[1:]))


def _interp_sorted(u, cdf, t):
    hi = torch.searchsorted(cdf, u, right=True)
    lo = (hi - 1).clamp(0, cdf.shape[-1] - 1)
    hi = hi.clamp(0, cdf.shape[-1] - 1)
    x0, x1, f0, f1 = cdf.gather(-1, lo), cdf.gather(-1, hi), t.gather(-1, lo), t.gather(-1, hi)
    return f0 + _clamp01(torch.nan_to_num((u - x0) / (x1 - x0), 0.0)) * (f1 - f0)


def _resample(sd, w, n, dilation):
    eps = float(np.finfo(np.float32).eps)
    if dilation > 0:
        pdf = w / (sd[:, 1:] - sd[:, :-1]).clamp_min(eps)
        t0, t1 = sd[:, :-1] - dilation, sd[:, 1:] + dilation
        posts = torch.sort(torch.cat([sd, t0, t1], -1), -1).values.clip(0, 1)
        best = torch.zeros_like(posts)
        for j in range(pdf.shape[-1]):
            inside = (t0[:, j:j + 1] <= posts) & (t1[:, j:j + 1] > posts)
            best = torch.where(inside, torch.maximum(best, pdf[:, j:j + 1]), best)
        wd = best[:, :-1] * (posts[:, 1:] - posts[:, :-1])
        wd = wd / wd.sum(-1, keepdim=True).clamp_min(eps)
        sd, w = posts[:, 1:-1], wd[:, 1:-1]
    prob = torch.softmax(torch.where(sd[:, 1:] > sd[:, :-1], torch.log(w), -math.inf), -1)
    cdf = torch.cumsum(prob[:, :-1], -1).clamp_max(1)
    z = torch.zeros_like(sd[:, :1])
    cdf = torch.cat([z, cdf, z + 1], -1)
    u = torch.linspace(1 / (2 * n), 1 - 1 / (2 * n) - eps, n, dtype=torch.float64, device=sd.device)
    c = _interp_sorted(u.expand(len(sd), n).contiguous(), cdf, sd)
    mid = (c[:, 1:] + c[:, :-1]) / 2
    first, last = 2 * c[:, :1] - mid[:, :1], 2 * c[:, -1:] - mid[:, -1:]
    return torch.cat([first.clamp_min(0), mid, last.clamp_max(1)], -1)


def _exact_sampling(case, s):
    o, d, near, far = (s[k].double() for k in ("o", "d", "near", "far"))
    R = len(o)
    sd = torch.tensor([[0.0, 1.0]], device=DEV, dtype=torch.float64).expand(R, 2)
    w = torch.ones(R, 1, device=DEV, dtype=torch.float64)
    res, prod = dict(density=[], weights=[]), 1
    for i in range(3):
        n = case["prop_samples"] if i < 2 else case["samples"]
        dilation = 0.0025 + 0.5 / prod
        prod *= n
        sd = _resample(sd, w, n, dilation if i else 0.0)
        td = sd * far[:, None] + (1 - sd) * near[:, None]
        if i == 2:
            return dict(res, sdist=sd, tdist=td)
        t = (td[:, 1:] + td[:, :-1]) / 2
        u = (_contract((d[:, None] * t[..., None] + o[:, None]).reshape(-1, 3)) + 1) / 2
        p = [v.detach().double() for v in _net_params(s["nets"][i])]
        dens = _layers(_exact_features(u, s["nets"][i].encoder, p[0]), p).reshape(R, n)
        tau = dens * (td[:, 1:] - td[:, :-1]) * d.norm(dim=-1, keepdim=True)
        trans = torch.exp(-torch.cat([torch.zeros_like(tau[:, :1]), torch.cumsum(tau[:, :-1], 1)], 1))
        w = -torch.expm1(-tau) * trans
        res["density"].append(dens)
        res["weights"].append(w)
    return res


def exact(case, seed):
    s, op = _inputs(case, seed), case["op"]
    curves = case.get("kinds") in ("curves", "all")
    chunk = 3_000_000 if curves else 6_000_000
    if op == "render":
        s["cast"] = case["cast"]
        if not case["grad"]:
            with torch.no_grad():
                return _exact_render(s, True, False, False, 4 * chunk)
        res = _exact_render(s, True, True, not case["cast"], chunk)
        del res["grad_delta"]
        return res
    if op == "field":
        return _exact_field(case, s)
    if op == "batch":
        got = [_exact_render(q, True, True, True, chunk) for q in s["scenes"]]
        return {k: torch.cat([q[k] for q in got]) for k in got[0]}
    if op == "operators":
        return _exact_operators(case, s)
    with torch.no_grad():
        if op == "grid":
            return _exact_grid(s)
        if op == "sampling":
            return _exact_sampling(case, s)
    return _exact_density(s)
