"""The work this framework is used for, as timed cases: the stages of the thin-shell pipeline
(octree, shell samples, signed distance, fit, dense field, marching cubes), the solvers beside the
learned fit, the share network's training step, and one whole pipeline call.

Sizes: the (3,5) torus-knot tube of 1,048,576 faces at octree resolution 256 with marching cubes at
512^3 (bench.py's default workload), the 10,240-face sphere at resolution 32 with a 128^3 grid (the
small workload), the uneven multi-mesh mix, and tubes and tori in between.

The octree's resolution is res (its depth is log2(res) + 1); the tube has rings x segs quads.
"""
import ctypes
import math

import numpy as np
import torch

from its_b200 import (OP_FP32_VALUES, OP_FP64, PREC_FP64, PREC_MIXED, STOP_RESIDUAL, Context, Operator, Svo, lib, meshes,
                      model_to_unit_cube, sharenet, uniform_bbox)
from its_b200.api import ShareNet, fit_residual_batch, learned_fit, learned_start_batch

TOL = 1e-6  # the fit's relative residual in every workload


def listed():
    return [
        # the smallest call of the path: the octree of the 10,240-face sphere
        {"name": "octree_small", "kind": "octree", "shape": "sphere", "faces": 10240, "res": 32},
        # the samples of the benchmark tube: a million triangles against the fine nodes and edges
        {"name": "samples_tube", "kind": "samples", "shape": "knot", "faces": 1048576, "res": 256},
        # the fit's right-hand side: tree over a million triangles, a query per corner vertex
        {"name": "distance_tube", "kind": "distance", "shape": "knot", "faces": 1048576, "res": 256},
        # the headline fit, repeated on a resident octree (a user refitting new right-hand sides)
        {"name": "fit_tube", "kind": "fit", "shape": "knot", "faces": 1048576, "res": 256},
        # the reference's method on the same tube: assembly and FP64 least-squares CG from zero
        {"name": "lscg_tube", "kind": "lscg", "shape": "knot", "faces": 1048576, "res": 256, "precision": "fp64"},
        # many meshes of uneven size fitted together: learned starts and their residuals
        {"name": "fit_batch", "kind": "batch", "meshes": 24, "fmin": 2000, "fmax": 60000},
        # the marching-cubes field, bit-exact form, twice the octree's resolution
        {"name": "field_512", "kind": "field", "shape": "knot", "faces": 1048576, "res": 256, "grid": 512, "mode": "fp64"},
        # the batch workload's field: the grid of a mesh is no finer than its octree
        {"name": "field_256", "kind": "field", "shape": "torus", "faces": 99000, "res": 256, "grid": 256, "mode": "fp64"},
        # case indices and triangle soup of a resident field
        {"name": "march_512", "kind": "march", "shape": "knot", "faces": 1048576, "res": 256, "grid": 512},
        # the cubic-basis workload's grid
        {"name": "cubic_128", "kind": "cubic", "shape": "sphere", "faces": 10240, "res": 32, "grid": 128},
        # one gradient of the share network at its training batch
        {"name": "train_step", "kind": "train", "rows": 65536},
        # the facade's call order end to end on a mesh of ordinary size, soups to the host
        {"name": "pipeline", "kind": "pipeline", "shape": "knot", "faces": 200000, "res": 128, "grid": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed kinds: face counts from 2,000 to a million with the octree resolution
    that such meshes are given, grids from half to twice (the field: four times) as fine, odd ones among them."""
    kind = rng.choice(["octree", "samples", "distance", "fit", "lscg", "batch", "field", "march", "cubic", "train",
                       "pipeline"])
    if kind == "train":
        return {"kind": kind, "rows": 64 * _log(rng, 16, 1024)}
    if kind == "batch":
        fmin = _log(rng, 2000, 8000)
        return {"kind": kind, "meshes": rng.randint(3, 24), "fmin": fmin, "fmax": fmin * rng.randint(2, 7)}
    faces = _log(rng, 2000, 20000 if kind == "cubic" else 1000000)
    shape = rng.choice(["sphere", "knot", "torus"] if faces <= 200000 else ["knot", "torus"])
    res = 32 if faces < 5000 else 64 if faces < 20000 else 128 if faces < 150000 else 256
    if rng.random() < 0.3 and res < 256 and kind != "cubic":
        res *= 2
    case = {"kind": kind, "shape": shape, "faces": faces, "res": min(res, 64) if kind == "cubic" else res}
    if kind == "lscg":
        case["precision"] = rng.choice(["fp64", "mixed"])
    if kind == "field":
        case["mode"] = rng.choice(["fp64", "fp32", "fast", "fast32"])
        if case["mode"].startswith("fast"):
            case["grid"] = res * rng.choice([1, 2] if res == 256 else [1, 2, 4])
        else:
            case["grid"] = rng.randint(res // 2, 2 * res)
    if kind == "march":
        case["grid"] = rng.choice([rng.randint(res // 2, 2 * res), res, 2 * res])
    if kind == "cubic":
        case["grid"] = rng.randint(res, 128)
    if kind == "pipeline":
        case["grid"] = res if res == 256 else res * rng.choice([1, 2])
    return case


# ---- inputs ------------------------------------------------------------------------------------

_shared = {}


def _context():
    """A program's one context, and the trained share network on it."""
    if not _shared:
        _shared["ctx"] = Context(0)
        params, norm = sharenet.load()
        _shared["net"] = ShareNet(_shared["ctx"], batch=4096, params=params)
        _shared["norm"] = np.ascontiguousarray(norm, np.float32)
    return _shared["ctx"], _shared["net"], _shared["norm"]


def _mesh(case, seed):
    """A closed mesh of about case['faces'] faces in the unit cube: the seed sets its shape or its noise."""
    rng = np.random.default_rng(seed)
    faces = case["faces"]
    if case["shape"] == "knot":
        segs = max(8, int(round(math.sqrt(faces / 64.0))))
        rings = max(16, int(round(faces / (2.0 * segs))))
        V, F = meshes.torus_knot_tube(rings=rings, segs=segs, seed=seed)
    elif case["shape"] == "torus":
        R, r = rng.uniform(0.6, 0.9), rng.uniform(0.15, 0.25)
        segs = max(8, int(round(math.sqrt(faces / 2.0 * r / R))))
        rings = max(8, int(round(faces / (2.0 * segs))))
        V, F = meshes.torus_mesh(R, r, rings, segs)
        V = V + rng.normal(0.0, 2e-4, V.shape)
    else:
        freq = max(2, int(round(math.sqrt(faces / 10.0))))
        V, F = meshes.superquadric_mesh(rng.uniform(0.7, 1.3), rng.uniform(0.7, 1.3), freq=freq)
    return model_to_unit_cube(V), np.ascontiguousarray(F, np.int32)


def _capacity(res):
    """Entries of a buffer that holds any such mesh's corner vertices, for results of a size that the
    caller does not know before the octree is built (2 to 16 res^2 over these shapes)."""
    return 20 * res * res + 4096


def _buffer(rows, cols=None, dtype=torch.float64):
    return torch.zeros(rows if cols is None else (rows, cols), dtype=dtype, device="cuda")


def _octree(case, seed, state):
    ctx = state["ctx"]
    V, F = _mesh(case, seed)
    o, end, w = uniform_bbox(V)
    state.update(V=torch.from_numpy(V).cuda(), F=torch.from_numpy(F).cuda(), o=o, w=w, end=end, res=case["res"])
    torch.cuda.synchronize()
    state["svo"] = Svo(ctx, state["V"], state["F"], case["res"], o, w)


def _rhs(state):
    svo = state["svo"]
    b = torch.empty(svo.num_verts, dtype=torch.float64, device="cuda")
    state["b"] = state["ctx"].signed_distance(svo.vertex_positions_device(), state["V"], state["F"], out=b)


def _train_inputs(rows, seed):
    """Normalised features and targets with the distributions that the training data have."""
    g = torch.Generator().manual_seed(seed)
    X = torch.randn((rows, 64), generator=g)
    X[:, 46:] = 0.0  # the features beyond the 46 in use
    y = torch.tanh(X[:, :8].sum(1) * 0.3) + 0.05 * torch.randn(rows, generator=g)
    params = sharenet.init_params(seed)
    return X, y, params


def prepare(case, seed):
    ctx, net, norm = _context()
    state = {"kind": case["kind"], "ctx": ctx, "net": net, "norm": norm}
    kind = case["kind"]
    if kind == "train":
        X, y, params = _train_inputs(case["rows"], seed)
        state["X"], state["y"] = X.cuda(), y.cuda()
        state["trainee"] = ShareNet(ctx, batch=(case["rows"] + 127) // 128 * 128, params=params)
    elif kind == "batch":
        svos, bs, bufs, rng = [], [], [], np.random.default_rng(seed)
        for m in meshes.batch_meshes(case["meshes"], fmin=case["fmin"], fmax=case["fmax"]):
            V = model_to_unit_cube(m["V"] + rng.normal(0.0, 1e-3, m["V"].shape))
            o, _, w = uniform_bbox(V)
            Vd, Fd = torch.from_numpy(V).cuda(), torch.from_numpy(m["F"]).cuda()
            torch.cuda.synchronize()
            svos.append(Svo(ctx, Vd, Fd, m["res"], o, w))
            b = torch.empty(svos[-1].num_verts, dtype=torch.float64, device="cuda")
            bs.append(ctx.signed_distance(svos[-1].vertex_positions_device(), Vd, Fd, out=b))
            bufs.append(_buffer(_capacity(m["res"])))
        state.update(svos=svos, bs=bs, bufs=bufs, outs=[buf[:b.shape[0]] for buf, b in zip(bufs, bs)])
    elif kind in ("octree", "pipeline"):
        V, F = _mesh(case, seed)
        o, end, w = uniform_bbox(V)
        state.update(V=torch.from_numpy(V).cuda(), F=torch.from_numpy(F).cuda(), o=o, w=w, end=end, res=case["res"])
        cap = _capacity(case["res"])
        state["pos"] = _buffer(cap, 3)
        if kind == "octree":
            state["own"] = _buffer(cap, dtype=torch.int32)
        else:
            R = state["grid"] = case["grid"]
            state.update(b=_buffer(cap), lam=_buffer(cap), soups=[np.zeros((12 * R * R + 1024, 3)) for _ in range(3)])
    else:
        _octree(case, seed, state)
        if kind == "samples":
            state["points"] = _buffer(2 * state["F"].shape[0] + state["V"].shape[0] + 1024, 3)
        if kind == "distance":
            state["P"] = state["svo"].vertex_positions_device()
            state["buf"] = _buffer(_capacity(case["res"]))
            state["out"] = state["buf"][:state["svo"].num_verts]
        elif kind in ("fit", "lscg"):
            _rhs(state)
            state["buf"] = _buffer(_capacity(case["res"]))
            state["out"] = state["buf"][:state["svo"].num_verts]
            state["mixed"] = case.get("precision") == "mixed"
        elif kind == "cubic":
            # coefficients of the size that cubic fits have: the field's own values, perturbed
            _rhs(state)
            g = torch.Generator().manual_seed(seed)
            state["lam"] = state["b"] * (1.0 + 0.1 * torch.randn(state["b"].shape, generator=g, dtype=torch.float64).cuda())
            state["grid"] = case["grid"]
            state["out"] = torch.empty((case["grid"] + 1) ** 3, dtype=torch.float64, device="cuda")
        elif kind in ("field", "march"):
            _rhs(state)
            lam = torch.empty_like(state["b"])
            learned_fit(state["svo"], net, state["b"], norm, TOL, out=lam)
            R = case["grid"]
            mode = case.get("mode", "fast")
            field = torch.empty((R + 1) ** 3, dtype=torch.float32 if mode.endswith("32") else torch.float64, device="cuda")
            state.update(lam=lam, grid=R, mode=mode, field=field)
            if kind == "march":
                state["svo"].eval_grid_fast(lam, state["o"], state["w"], R, out=field)
                state["cube"] = torch.empty(R ** 3, dtype=torch.uint8, device="cuda")
                state["tri"] = _buffer(12 * R * R + 1024, 3)
    torch.cuda.synchronize()
    return state


# ---- one pass ----------------------------------------------------------------------------------


def _ptr(a):
    return ctypes.c_void_p(a.data_ptr() if isinstance(a, torch.Tensor) else a.ctypes.data)


def _vertices(svo, pos, own):
    svo.ctx.check(lib().its_svo_get_vertices(svo.h, _ptr(pos), None if own is None else _ptr(own)), "its_svo_get_vertices")


def _samples(svo, s, out):
    n, on_edges = ctypes.c_int64(0), ctypes.c_int64(0)
    svo.ctx.check(lib().its_shell_samples(svo.h, _ptr(s["V"]), s["V"].shape[0], _ptr(s["F"]), s["F"].shape[0], _ptr(out),
                                          out.shape[0], ctypes.byref(n), ctypes.byref(on_edges)), "its_shell_samples")
    return n.value, on_edges.value


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "octree":
        svo = Svo(ctx, s["V"], s["F"], s["res"], s["o"], s["w"])
        _vertices(svo, s["pos"], s["own"])
        return {"vertices": s["pos"], "owners": s["own"], "voxels": svo.num_voxels, "nodes": svo.num_nodes,
                "corners": svo.num_verts, "edges": svo.num_edges}
    if kind == "samples":
        count, on_edges = _samples(s["svo"], s, s["points"])
        return {"points": s["points"], "count": count, "on_edges": on_edges}
    if kind == "distance":
        ctx.signed_distance(s["P"], s["V"], s["F"], out=s["out"])
        return s["buf"]
    if kind == "fit":
        _, rep = learned_fit(s["svo"], s["net"], s["b"], s["norm"], TOL, out=s["out"])
        return {"lambda": s["buf"], "converged": rep["converged"], "iterations": rep["iterations"]}
    if kind == "lscg":
        op = Operator(s["svo"], mode=OP_FP32_VALUES if s["mixed"] else OP_FP64)
        _, rep = op.solve(s["b"], tol=TOL, stop_rule=STOP_RESIDUAL, precision=PREC_MIXED if s["mixed"] else PREC_FP64,
                          out=s["out"])
        op.close()
        return {"lambda": s["buf"], "converged": rep["converged"], "iterations": rep["iterations"]}
    if kind == "batch":
        lams = learned_start_batch(s["svos"], s["net"], s["bs"], s["norm"], outs=s["outs"])
        rel = fit_residual_batch(s["svos"], s["bs"], lams)
        return {"lambdas": s["bufs"], "converged": (rel <= TOL).astype(np.int32)}
    if kind == "field":
        svo, mode = s["svo"], s["mode"]
        if mode == "fp64":
            return svo.eval_grid(s["lam"], s["o"], s["w"], s["grid"], out=s["field"])
        if mode == "fp32":
            return svo.eval_grid_f32(s["lam"], s["o"], s["w"], s["grid"], out=s["field"])
        return svo.eval_grid_fast(s["lam"], s["o"], s["w"], s["grid"], out=s["field"], fp32=mode == "fast32")
    if kind == "march":
        n = ctypes.c_int64(0)
        ctx.check(lib().its_marching_cubes(ctx.h, _ptr(s["field"]), s["grid"], _ptr(s["o"]), _ptr(s["w"]), 0.0,
                                           _ptr(s["cube"]), _ptr(s["tri"]), s["tri"].shape[0], ctypes.byref(n)),
                  "its_marching_cubes")
        return {"cases": s["cube"], "soup": s["tri"], "vertices": n.value}
    if kind == "cubic":
        return s["svo"].eval_grid_cubic(s["lam"], s["o"], s["w"], s["grid"], out=s["out"])
    if kind == "train":
        grad, loss = s["trainee"].gradient(s["X"], s["y"])
        return {"gradient": grad, "loss": loss}
    # the facade's order: octree, samples, right-hand side, fit, iso levels, field and marching cubes
    svo = Svo(ctx, s["V"], s["F"], s["res"], s["o"], s["w"])
    n = svo.num_verts
    count, _ = _samples(svo, s, pts := torch.empty((2 * s["F"].shape[0] + s["V"].shape[0] + 1024, 3),
                                                   dtype=torch.float64, device="cuda"))
    _vertices(svo, s["pos"], None)
    b, lam = s["b"][:n], s["lam"][:n]
    ctx.signed_distance(s["pos"][:n], s["V"], s["F"], out=b)
    learned_fit(svo, s["net"], b, s["norm"], TOL, out=lam)
    inner, outer, _ = svo.shell_iso_values(lam, torch.cat([s["V"], pts[:count]]))
    isos, cap, cnt = np.array([outer, inner, 0.0]), np.full(3, s["soups"][0].shape[0], np.int64), np.zeros(3, np.int64)
    soups = (ctypes.c_void_p * 3)(*[x.ctypes.data for x in s["soups"]])
    ctx.check(lib().its_eval_grid_mc(svo.h, _ptr(lam), _ptr(s["o"]), _ptr(s["w"]), s["grid"], 1, _ptr(isos), 3, soups,
                                     _ptr(cap), _ptr(cnt)), "its_eval_grid_mc")
    return {"lambda": s["lam"], "b": s["b"], "inner": inner, "outer": outer, "soups": s["soups"], "counts": cnt}


# ---- what a pass cannot do without -------------------------------------------------------------


def work(case):
    """Bytes in and out and the arithmetic of the method, with the unknowns of such surfaces taken as
    3 res^2 and 51 entries per row (the benchmark tube: 196,681 and 50.9)."""
    kind = case["kind"]
    if kind == "train":
        B = case["rows"]
        return {"bytes": 4.0 * (B * 65 + 2 * 41345), "flops": 6.0 * B * 41088}
    if kind == "batch":
        faces = case["meshes"] * (case["fmax"] - case["fmin"]) / math.log(case["fmax"] / case["fmin"])
        n = 2.0 * faces
        return {"bytes": 16.0 * n, "flops": 2.0 * 41088 * n / 6 + 40.0 * n}
    F, res = case["faces"], case["res"]
    n = 3.0 * res * res
    mesh = 24.0 * F  # three indices a face, half a vertex a face
    R = case.get("grid", 0)
    pts, vox = (R + 1.0) ** 3, float(R) ** 3
    depth = math.log2(res) + 1
    if kind == "octree":
        return {"bytes": mesh + 24.0 * n + 136.0 * n, "flops": 100.0 * F}
    if kind == "samples":
        return {"bytes": mesh + 24.0 * 0.9 * F, "flops": 100.0 * F}
    if kind == "distance":
        return {"bytes": mesh + 32.0 * n, "flops": 100.0 * F + 2000.0 * n}
    if kind == "fit":
        return {"bytes": 24.0 * n, "flops": 2.0 * 41088 * n / 6 + 40.0 * n}
    if kind == "lscg":
        return {"bytes": 16.0 * n, "flops": 4.0 * 51 * n * 31}
    if kind == "field":
        size = 4.0 if case["mode"].endswith("32") else 8.0
        return {"bytes": size * pts + 8.0 * n, "flops": (3.0 * 33 if case["mode"].startswith("fp") else 4.0) * pts}
    if kind == "march":
        return {"bytes": 8.0 * pts + vox + 24.0 * 5 * R * R, "flops": pts}
    if kind == "cubic":
        return {"bytes": 8.0 * pts + 8.0 * n, "flops": 20.0 * depth * pts}
    return {"bytes": mesh + 200.0 * n + 8.0 * pts + 3 * (8.0 * pts + 24.0 * 5 * R * R),
            "flops": 300.0 * F + 2000.0 * n + 2.0 * 41088 * n / 6}


def exact(case, seed):
    """The share network's loss and gradient in 64 bits; the other kinds' outputs are whole numbers or
    follow from the octree, which only this package builds."""
    if case["kind"] != "train":
        return None
    X, y, params = _train_inputs(case["rows"], seed)
    X, y = X.double().cuda(), y.double().cuda()
    P = torch.from_numpy(params).double().cuda().requires_grad_(True)
    h, at = X, 0
    for rows, cols in ((128, 64), (128, 128), (128, 128)):
        W, bias = P[at:at + rows * cols].view(rows, cols), P[at + rows * cols:at + rows * cols + rows]
        at += rows * cols + rows
        h = torch.nn.functional.gelu(h @ W.T + bias, approximate="tanh")
    out = h @ P[at:at + 128] + P[at + 128]
    loss = ((out - y) ** 2).mean()
    loss.backward()
    return {"gradient": P.grad, "loss": float(loss.detach())}
