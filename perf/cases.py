"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the package's public entry points: one octree leaf
meshed on the GPU or into host arrays, a whole span meshed on the GPU or into
pinned memory, dual contouring, batches of uneven spans, point batches of the
estimator in its forms, gradients, a differentiable estimator step and a step
of the depth-map fit.  Sizes are those of the benchmark and the tests: leaves
of 64 cells per axis (cantucci's), spans up to 512, batches of spans of 8 to
64 cells, up to a few million points, depth maps up to 1024 x 1024.
"""
import math

import numpy as np
import torch

import cantucci_gb300 as cg
from cantucci_gb300 import autograd as cg_autograd
from cantucci_gb300 import fit as cg_fit
from cantucci_gb300.batch import BatchMesher

BAILOUT = 2.5


def listed():
    return [
        # An octree leaf as ShapeMesh requests it, left on the GPU for drawing: the
        # call whose latency a camera move waits for.
        {"name": "leaf_device", "kind": "mesh", "res": 64, "edge": 0.3, "power": 8, "iters": 15,
         "placement": "centroid", "normals": "fd"},
        # The same leaf into host arrays that a pool thread keeps: the reference's own
        # call (generate_for_box).
        {"name": "leaf_host", "kind": "mesh_host", "res": 64, "edge": 0.3, "power": 8, "iters": 15},
        # The whole bulb at the benchmark's resolution, on the GPU.
        {"name": "span_512", "kind": "mesh", "res": 512, "edge": 2.4, "power": 8, "iters": 15,
         "placement": "centroid", "normals": "fd"},
        # A whole span for export, into pinned host memory.
        {"name": "span_pinned_256", "kind": "mesh_pinned", "res": 256, "edge": 2.4, "power": 8,
         "iters": 15},
        # Dual contouring with analytic normals: the sharper mesh of the same bulb.
        {"name": "span_contoured_256", "kind": "mesh", "res": 256, "edge": 2.4, "power": 8,
         "iters": 15, "placement": "qef", "normals": "analytic"},
        # All leaves that a frame of the level-of-detail driver asks for, and many
        # more: uneven spans in one replayed graph.
        {"name": "batch_p8", "kind": "batch", "spans": 4096, "power": 8, "iters": 15,
         "graph": True},
        # A batch of the generic power (trigonometric form), launched directly.
        {"name": "batch_p6", "kind": "batch", "spans": 512, "power": 6, "iters": 10,
         "graph": False},
        # The smallest call: a handful of probes of the estimator.
        {"name": "points_small", "kind": "points", "n": 1021, "form": "p8", "power": 8.0,
         "iters": 15, "fast": False},
        # A large, odd point batch of the rotated real-power form.
        {"name": "points_polar", "kind": "points", "n": 3000017, "form": "polar", "power": 8.3,
         "iters": 15, "fast": False},
        # Shading normals of points on the surface band, forward mode.
        {"name": "normals_band", "kind": "normals", "n": 1500001, "power": 8.0, "iters": 15,
         "with_power": False},
        # A training step on the differentiable estimator: forward and backward.
        {"name": "estimator_step", "kind": "estimator", "n": 1000003, "power": 8.0, "iters": 15},
        # One step of fitting power and rotation to a depth map.
        {"name": "fit_step_512", "kind": "fit", "width": 512, "height": 512, "power": 8.3,
         "fast": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mesh", "mesh", "mesh_host", "mesh_pinned", "batch", "points", "points",
                       "normals", "estimator", "fit"])
    power = rng.choice([8, 8, 8, 6, 10])
    iters = rng.choice([10, 15, 15, 20])
    if kind == "mesh":
        placement = rng.choice(["centroid", "centroid", "qef"])
        return {"kind": kind, "res": rng.choice([16, 32, 64, 128, 256]),
                "edge": round(rng.uniform(0.1, 2.4), 3), "power": power, "iters": iters,
                "placement": placement, "normals": rng.choice(["fd", "analytic"])}
    if kind == "mesh_host":
        return {"kind": kind, "res": rng.choice([16, 32, 64, 128]),
                "edge": round(rng.uniform(0.05, 2.4), 3), "power": power, "iters": iters}
    if kind == "mesh_pinned":
        return {"kind": kind, "res": rng.choice([64, 128, 256]),
                "edge": round(rng.uniform(0.5, 2.4), 3), "power": power, "iters": iters}
    if kind == "batch":
        return {"kind": kind, "spans": _log_int(rng, 4, 1024), "power": power, "iters": iters,
                "graph": rng.random() < 0.5}
    if kind == "points":
        form = rng.choice(["p8", "int", "polar"])
        p = {"p8": 8.0, "int": float(rng.choice([6, 10])),
             "polar": round(rng.uniform(6.0, 10.0), 2)}[form]
        return {"kind": kind, "n": _log_int(rng, 500, 3000000), "form": form, "power": p,
                "iters": iters, "fast": rng.random() < 0.3}
    if kind == "normals":
        return {"kind": kind, "n": _log_int(rng, 1000, 1500000),
                "power": round(rng.uniform(7.5, 8.5), 2), "iters": rng.choice([10, 15]),
                "with_power": rng.random() < 0.5}
    if kind == "estimator":
        return {"kind": kind, "n": _log_int(rng, 1000, 1000000),
                "power": round(rng.uniform(7.5, 8.5), 2), "iters": rng.choice([10, 15])}
    w = rng.choice([128, 200, 256, 333, 512])
    return {"kind": "fit", "width": w, "height": rng.choice([w, 3 * w // 4]),
            "power": round(rng.uniform(7.8, 8.4), 2), "fast": rng.random() < 0.7}


# ---- inputs ---------------------------------------------------------------

def _rng(seed):
    return np.random.default_rng(1000003 * int(seed) + 17)


def _span(case, seed):
    """A span of the given edge: around the origin if it takes in the whole
    bulb, else centred on a point of the surface, where a ray from outside
    comes to rest."""
    rng = _rng(seed)
    e = float(case["edge"])
    if e > 1.5:
        c = rng.uniform(-0.02, 0.02, size=3)
    else:
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        t = 1.4
        for _ in range(60):
            p = torch.tensor((t * d)[None], dtype=torch.float64)
            step = float(_plain_estimator(p, case["power"], case["iters"], case["power"] == 8)[0])
            t -= max(step, 0.0)
            if step < 2e-3 or t < 0.5:
                break
        c = t * d
    half = e / 2.0
    return cg.Span((c - half).astype(np.float32), (c + half).astype(np.float32))


def _uneven_spans(n, seed):
    """Spans centred on the shell of radius 0.8 to 1.15, edges 2^-3 to 2^-7, of
    8, 16, 32 or 64 cells per axis (the same list of resolutions for every seed)."""
    res = _rng(n).choice(np.array([8, 16, 32, 64], np.uint32), size=n)
    rng = _rng(seed)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    c = (d * rng.uniform(0.8, 1.15, size=(n, 1))).astype(np.float32)
    half = np.ldexp(np.float32(0.5), -rng.integers(3, 8, size=n)).astype(np.float32)[:, None]
    return np.concatenate([c - half, c + half], axis=1).astype(np.float32), res


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(7919 * int(seed) + 3)


def _uniform_points(n, seed):
    return torch.rand((n, 3), generator=_generator(seed), device="cuda") * 2.4 - 1.2


def _power(case, seed):
    """The case's real power moved a little by the seed, as f32."""
    return float(np.float32(case["power"] + _rng(seed).uniform(-0.05, 0.05)))


def _angles(seed):
    return [float(np.float32(v)) for v in _rng(seed + 1).uniform(-0.3, 0.3, size=3)]


def _rotation(angles, like):
    a, b, c = angles
    ca, sa, cb, sb, cc, sc = (math.cos(a), math.sin(a), math.cos(b), math.sin(b), math.cos(c),
                              math.sin(c))
    m = [[cc * cb, cc * sb * sa - sc * ca, cc * sb * ca + sc * sa],
         [sc * cb, sc * sb * sa + cc * ca, sc * sb * ca - cc * sa],
         [-sb, cb * sa, cb * ca]]
    return torch.tensor(m, dtype=like.dtype, device=like.device)


def _plain_estimator(p, power, iters, polynomial):
    """The estimator in plain torch, in p's own precision.  `polynomial`: the
    reference's power-8 polynomial, else the polar map."""
    z, dr = p.clone(), torch.ones_like(p[:, 0])
    r = torch.zeros_like(dr)
    live = torch.ones_like(dr, dtype=torch.bool)
    for _ in range(iters):
        x, y, w = z[:, 0], z[:, 1], z[:, 2]
        r = torch.where(live, torch.sqrt(x * x + y * y + w * w), r)
        live = live & ~(r > BAILOUT)
        dr = torch.where(live, r ** (power - 1) * power * dr + 1, dr)
        if polynomial:
            x2, y2, z2 = x * x, y * y, w * w
            q = x2 + y2
            a = 1 + (z2 ** 4 - 28 * z2 ** 3 * q + 70 * z2 ** 2 * q ** 2 - 28 * z2 * q ** 3) / q ** 4
            n = torch.stack([
                a * (x2 ** 4 - 28 * x2 ** 3 * y2 + 70 * x2 ** 2 * y2 ** 2 - 28 * x2 * y2 ** 3
                     - y2 ** 4),
                8 * a * x * y * (x2 ** 3 - 7 * x2 ** 2 * y2 + 7 * x2 * y2 ** 2 - y2 ** 3),
                8 * w * torch.sqrt(q) * (z2 - q) * (z2 ** 2 - 6 * z2 * q + q ** 2)], 1)
        else:
            th = torch.acos((w / r).clamp(-1, 1)) * power
            ph = torch.atan2(y, x) * power
            k = r ** power
            n = torch.stack([k * torch.sin(th) * torch.cos(ph), k * torch.sin(ph) * torch.sin(th),
                             k * torch.cos(th)], 1)
        z = torch.where(live[:, None], n + p, z)
    return 0.5 * torch.log(r) * r / dr


def _band_points(n, seed, power, iters):
    """n points on the surface band |DE| < 1e-3: uniform in the cube, moved by
    8 sphere-trace steps along random directions."""
    g = _generator(seed)
    kept, have = [], 0
    while have < n:
        m = max(4096, min(4 * n, 4000000))
        p = torch.rand((m, 3), generator=g, device="cuda") * 2.4 - 1.2
        d = torch.randn((m, 3), generator=g, device="cuda")
        d = d / d.norm(dim=1, keepdim=True)
        for _ in range(8):
            p = p + d * _plain_estimator(p, power, iters, False)[:, None]
        e = _plain_estimator(p, power, iters, False)
        kept.append(p[torch.isfinite(e) & (e.abs() < 1e-3)])
        have += kept[-1].shape[0]
    return torch.cat(kept)[:n].contiguous()


def _vertex_room(res):
    """More vertices than the surface has in a span of `res` cells per axis."""
    return min(res ** 3, 24 * res * res + 4096)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("mesh", "mesh_host", "mesh_pinned"):
        s = {"case": case, "span": _span(case, seed), "mesher": cg.Mesher(),
             "shape": cg.Mandelbulb(case["power"], case["iters"], BAILOUT)}
        room = _vertex_room(case["res"])
        if kind == "mesh":
            s["mesher"].set_placement(case["placement"])
            s["mesher"].set_normals(case["normals"])
            s["vertices"] = torch.zeros((room, 7), dtype=torch.float32, device="cuda")
            s["indices"] = torch.zeros(8 * room, dtype=torch.int32, device="cuda")
        elif kind == "mesh_pinned":
            s["vertices"] = torch.zeros((room, 7), dtype=torch.float32, pin_memory=True)
            s["indices"] = torch.zeros(8 * room, dtype=torch.int32, pin_memory=True)
        else:
            s["vertices"] = np.zeros(room, cg.VERTEX_DTYPE)
            s["indices"] = np.zeros(8 * room, np.uint32)
        return s
    if kind == "batch":
        spans, res = _uneven_spans(case["spans"], seed)
        room = int(np.sum(np.minimum(res.astype(np.int64) ** 3, 8 * res.astype(np.int64) ** 2)))
        s = {"case": case, "batch": BatchMesher(spans, res, vertex_cap=room, index_cap=8 * room),
             "shape": cg.Mandelbulb(case["power"], case["iters"], BAILOUT)}
        # one run, so that the batch is planned (and its graph captured); its
        # buffers are cleared so that the room past the meshes reads 0
        out = s["batch"].run(s["shape"], graph=case["graph"])
        out.vertices.zero_()
        out.indices.zero_()
        return s
    if kind == "points":
        if case["form"] == "polar":
            shape = cg.MandelbulbPolar(_power(case, seed), case["iters"], BAILOUT, _angles(seed))
        else:
            shape = cg.Mandelbulb(int(case["power"]), case["iters"], BAILOUT)
        return {"case": case, "shape": shape.fast() if case["fast"] else shape,
                "points": _uniform_points(case["n"], seed)}
    if kind in ("normals", "estimator"):
        power = _power(case, seed)
        s = {"case": case, "power": power,
             "points": _band_points(case["n"], seed, power, case["iters"])}
        if kind == "estimator":
            s["weights"] = torch.randn(case["n"], generator=_generator(seed + 1), device="cuda")
            s["p"] = torch.tensor(power, requires_grad=True)
            s["rot"] = torch.zeros(3, requires_grad=True)
            s["points"].requires_grad_(True)
        return s
    cam = cg_fit.camera(case["width"], case["height"], 2.5, 60.0)
    target = cg_fit.render(_power(case, seed), _angles(seed), cam, fast=True)
    start = _rng(seed + 2)
    return {"case": case, "cam": cam, "target": target,
            "surface": cg_fit.surface_points(target, cam),
            "p": torch.tensor(case["power"] + float(start.uniform(-0.2, 0.2)), requires_grad=True),
            "rot": torch.tensor(start.uniform(-0.2, 0.2, size=3).astype(np.float32),
                                requires_grad=True)}


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "mesh":
        nv, ni, _ = s["mesher"].generate_device(s["span"], s["shape"], case["res"], s["vertices"],
                                                s["indices"], strict=False)
        return {"vertices": s["vertices"], "indices": s["indices"], "counts": [nv, ni]}
    if kind in ("mesh_host", "mesh_pinned"):
        _, _, nv, ni, _ = s["mesher"].generate(s["span"], s["shape"], case["res"],
                                               vertices=s["vertices"], indices=s["indices"],
                                               strict=False)
        v = s["vertices"]
        if kind == "mesh_host":
            v = v.view(np.float32).reshape(-1, 7)
        return {"vertices": v, "indices": s["indices"], "counts": [nv, ni]}
    if kind == "batch":
        out = s["batch"].run(s["shape"], graph=case["graph"])
        return {"vertices": out.vertices, "indices": out.indices, "results": out.results,
                "totals": out.totals}
    if kind == "points":
        return s["shape"].batch_min_distance_from(s["points"])
    if kind == "normals":
        g = cg_autograd.de_grad(s["points"], s["power"], max_iters=case["iters"], mode="tangent",
                                with_power=case["with_power"])
        return {"distance": g[:, 0], "gradient": g[:, 1:4], "power_rotation": g[:, 4:]}
    if kind == "estimator":
        d = cg_autograd.mandelbulb_de(s["points"], s["p"], s["rot"], case["iters"], BAILOUT)
        loss = (d * s["weights"]).sum()
        gp, gpow, grot = torch.autograd.grad(loss, [s["points"], s["p"], s["rot"]])
        return {"distance": d.detach(), "points_grad": gp, "power_grad": gpow,
                "rotation_grad": grot}
    depth = cg_fit.depth_render(s["p"], s["rot"], s["cam"], fast=case["fast"], cap=2.0)
    loss = cg_fit.l1_loss(depth, s["target"])
    loss = loss + cg_fit.surface_loss(s["p"], s["rot"], s["surface"], cap=1.0)
    gpow, grot = torch.autograd.grad(loss, [s["p"], s["rot"]])
    return {"depth": depth.detach(), "loss": loss.detach(), "power_grad": gpow,
            "rotation_grad": grot}


def exact(case, seed):
    """The distances of point batches in 64 bits.  Meshes follow the signs of
    the reference's 32-bit distances; distances on the surface band,
    derivatives and marches follow the chaotic map's 32-bit orbits: those have
    no 64-bit counterpart."""
    if case["kind"] != "points":
        return None
    p = _uniform_points(case["n"], seed).double()
    if case["form"] == "polar":
        p = p @ _rotation(_angles(seed), p)
        return _plain_estimator(p, _power(case, seed), case["iters"], False)
    return _plain_estimator(p, int(case["power"]), case["iters"], case["form"] == "p8")


# Operations of one loop step: the power-8 polynomial as the reference writes
# it, and the polar form with each transcendental function counted as 10.
_STEP_P8, _STEP_POLAR = 76, 100


def work(case):
    """Outputs (and point inputs) moved once; the estimator's operations at the
    mean step counts of the bulb (4 over the whole cube, 10 near the surface,
    13 at the vertices)."""
    kind = case["kind"]
    step = _STEP_P8 if int(round(case["power"])) == 8 and kind not in (
        "normals", "estimator", "fit") and case.get("form", "p8") == "p8" else _STEP_POLAR
    if kind in ("mesh", "mesh_host", "mesh_pinned"):
        res, cube = case["res"], case["edge"] > 1.5
        vertices = (14 if cube else 3) * res * res
        corners = (res + 1) ** 3
        return {"bytes": vertices * 52, "flops": step * ((4 if cube else 10) * corners
                                                         + 7 * 13 * vertices)}
    if kind == "batch":
        corners, vertices = 81000 * case["spans"], 3100 * case["spans"]
        return {"bytes": vertices * 52, "flops": step * (10 * corners + 7 * 13 * vertices)}
    if kind == "points":
        return {"bytes": 16 * case["n"], "flops": step * 4 * case["n"]}
    if kind == "normals":
        return {"bytes": 44 * case["n"], "flops": 2 * step * 13 * case["n"]}
    if kind == "estimator":
        return {"bytes": 36 * case["n"], "flops": 3 * step * 13 * case["n"]}
    pixels = case["width"] * case["height"]
    return {"bytes": 12 * pixels, "flops": step * pixels * (50 + 2 * 13)}
