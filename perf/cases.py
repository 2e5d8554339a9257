"""Workloads of the KIFMM evaluator, each called as a user's program calls it.

Kinds of case:

solve     one solve with the points on the GPU, as an iterative solver or a
          time step calls it on a tree it keeps: new densities in
          (kfmm_set_sources_device), kfmm_run, potentials out
          (kfmm_get_potentials_device).  The tree, the plan and the target
          upload belong to the geometry and are prepared once.
evaluate  the drop-in `run`: kfmm_evaluate on pinned host arrays, host
          densities and points in, host potentials out.
batch     many small solves of uneven size under one CUDA graph: new
          densities for each, one launch, each solve's potentials out.
direct    the reference's own check: the exact sum at sampled targets over
          all sources (kfmm_direct_evaluation).
mlp       training steps of the leaf-size cost model (kfmm_mlp_train): forward,
          backward and Adam from given parameters.

Sizes, leaf sizes and NP are those of the benchmark configurations and the
tests (65,536 points at NP 4 and 128 per leaf, 1,048,576 and 4,194,304 at NP 6
and 512, 4,194,304 on the ellipsoid surface at NP 4 and 256, batches of 4,096 to
262,144 at NP 3 and 4), with small and ragged ones beside them.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "kifmm--hybrid--double-only_b200")


def _package():
    """The package directory (its name is no identifier) under the name kifmm_b200."""
    if "kifmm_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("kifmm_b200", os.path.join(_PKG, "__init__.py"),
                                                      submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["kifmm_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["kifmm_b200"]


def _solve(name, dist, n, ppb, np_, prec, coincide=0):
    return {"name": name, "kind": "solve", "dist": dist, "n": n, "ppb": ppb, "np": np_,
            "prec": prec, "coincide": coincide}


def listed():
    return [
        # a small solve inside a larger program: launches and latency count
        _solve("solve_4k_np4_fp64", "uniform", 4096, 64, 4, "fp64"),
        # a small ragged cloud on a deep adaptive tree (W and X lists)
        _solve("solve_20k_np3_ellipse_mixed", "ellipseUniformAngles", 20011, 32, 3, "mixed"),
        # the configuration the reference's CPU build is run on, sources = targets
        _solve("solve_65k_np4_fp64", "uniform", 65536, 128, 4, "fp64", 1),
        # the highest accuracy, a ragged size
        _solve("solve_100k_np8_fp64", "uniform", 100003, 250, 8, "fp64"),
        # the medium configuration, mixed form
        _solve("solve_1m_np6_mixed", "uniform", 1048576, 512, 6, "mixed"),
        # the large non-uniform configuration: a surface, densities of both signs
        _solve("solve_4m_np4_ellipsoid_mixed", "ellipsoidSurface", 4194304, 256, 4, "mixed"),
        # the headline configuration in both forms
        _solve("solve_4m_np6_mixed", "uniform", 4194304, 512, 6, "mixed"),
        _solve("solve_4m_np6_fp64", "uniform", 4194304, 512, 6, "fp64"),
        # many small solves in one graph (a smaller draw of the batched configuration)
        {"name": "batch_32_mixed", "kind": "batch", "count": 32, "nmin": 4096, "nmax": 262144,
         "mix": 2024, "prec": "mixed"},
        # the drop-in evaluator's call, host arrays to host potentials
        {"name": "evaluate_1m_np6_fp64", "kind": "evaluate", "dist": "uniform", "n": 1048576,
         "ppb": 512, "np": 6, "prec": "fp64", "coincide": 0},
        # the accuracy check that every run of the driver ends with
        {"name": "direct_1000x1m", "kind": "direct", "nt": 1000, "ns": 1048576},
        # refitting the cost model on the harvested measurements
        {"name": "mlp_train_20k", "kind": "mlp", "F": 73, "H": 64, "O": 5, "B": 19200, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# leaf sizes in use at each NP
_PPB = {3: (48, 160), 4: (48, 256), 5: (64, 320), 6: (64, 512), 7: (96, 512), 8: (128, 512)}
_DISTS = ("uniform", "uniform", "ellipseUniformAngles", "ellipsoidSurface")


def draw(rng):
    kind = rng.choices(("solve", "evaluate", "batch", "direct", "mlp"), (60, 12, 10, 10, 8))[0]
    if kind in ("solve", "evaluate"):
        np_ = rng.choices((3, 4, 5, 6, 7, 8), (2, 4, 1, 4, 1, 1))[0]
        prec = rng.choice(("mixed", "fp64"))
        return {"kind": kind, "dist": rng.choice(_DISTS),
                "n": _log(rng, 4096, 2097152 if prec == "mixed" and kind == "solve" else 1048576),
                "ppb": _log(rng, *_PPB[np_]), "np": np_, "prec": prec,
                "coincide": rng.choice((0, 0, 1))}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(8, 32), "nmin": 4096,
                "nmax": _log(rng, 16384, 262144), "mix": rng.randrange(1 << 30),
                "prec": rng.choice(("mixed", "mixed", "fp64"))}
    if kind == "direct":
        return {"kind": kind, "nt": _log(rng, 100, 3000), "ns": _log(rng, 65536, 1048576)}
    return {"kind": kind, "F": rng.randint(40, 96), "H": 64, "O": rng.randint(3, 8),
            "B": _log(rng, 1000, 19200), "steps": rng.randint(2, 10)}


def _precision(K, case):
    return K.MIXED if case["prec"] == "mixed" else K.PLAIN_FP64


def _handle():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


_SRC = ("sx", "sy", "sz", "den")
_TRG = ("tx", "ty", "tz")


class _OnDevice:
    """A plan and its points on the GPU, with room for the potentials."""

    def __init__(self, K, plan, pts):
        self.K, self.plan = K, plan
        self.src = [torch.from_numpy(pts[k]).cuda() for k in _SRC]
        self.trg = [torch.from_numpy(pts[k]).cuda() for k in _TRG]
        self.pot = torch.empty(plan.nt, dtype=torch.float64, device="cuda")
        K.check(K.lib().kfmm_set_targets_device(plan.handle, *[t.data_ptr() for t in self.trg],
                                                _handle()), "set_targets_device")

    def set_sources(self, stream):
        self.K.check(self.K.lib().kfmm_set_sources_device(
            self.plan.handle, *[t.data_ptr() for t in self.src], stream), "set_sources_device")

    def potentials(self, stream):
        self.K.check(self.K.lib().kfmm_get_potentials_device(
            self.plan.handle, self.pot.data_ptr(), stream), "get_potentials_device")
        return self.pot


def _batch_specs(case, seed):
    from kifmm_b200 import batched
    sp = batched.specs(case["count"], nmin=case["nmin"], nmax=case["nmax"], seed=case["mix"])
    return [{**s, "seed": (seed * 1009 + i) % (1 << 31)} for i, s in enumerate(sp)]


def _check_points(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    def draw_(n, lo):
        return lo + (1.0 - lo) * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    src = [draw_(case["ns"], -1.0) for _ in range(3)] + [draw_(case["ns"], 0.0)]
    return src, [draw_(case["nt"], -1.0) for _ in range(3)]


def _mlp_data(case, seed):
    """Standardised features, log-time targets that depend on them, and the
    usual starting parameters."""
    rng = np.random.default_rng(seed)
    F, H, O, B = case["F"], case["H"], case["O"], case["B"]
    X = rng.standard_normal((B, F)).astype(np.float32)
    T = (np.tanh(X @ rng.standard_normal((F, O)) / math.sqrt(F)) - 1.0
         + 0.1 * rng.standard_normal((B, O))).astype(np.float32)
    p = np.concatenate([a for fi, fo in ((F, H), (H, H), (H, O))
                        for a in (rng.normal(0, math.sqrt(2.0 / fi), fi * fo), np.zeros(fo))])
    return X, T, p.astype(np.float32)


def prepare(case, seed):
    K = _package()
    kind = case["kind"]
    if kind in ("solve", "evaluate"):
        pts = K.generate_points(case["n"], case["dist"], case["coincide"], seed)
        tree = K.Tree(*[pts[k] for k in ("sx", "sy", "sz", "tx", "ty", "tz")], case["ppb"],
                      device=True)
        plan = K.Plan(tree, case["np"], _precision(K, case))
        if kind == "solve":
            return {"kind": kind, "K": K, "tree": tree, "one": _OnDevice(K, plan, pts)}
        pinned = {k: torch.from_numpy(pts[k]).pin_memory().numpy() for k in _SRC + _TRG}
        out = torch.empty(case["n"], dtype=torch.float64).pin_memory().numpy()
        return {"kind": kind, "K": K, "tree": tree, "plan": plan, "pts": pinned, "pot": out}
    if kind == "batch":
        from kifmm_b200 import autotune, batched
        table = autotune.ConfigTable(os.path.join(_PKG, "tuning_data", "b200_batched_configs.json"))
        b = batched.BatchedSolves(K, _batch_specs(case, seed), _precision(K, case), table)
        return {"kind": kind, "K": K, "batch": b,
                "each": [_OnDevice(K, s["plan"], s["pts"]) for s in b.solves]}
    if kind == "direct":
        src, trg = _check_points(case, seed)
        return {"kind": kind, "K": K, "src": src, "trg": trg,
                "pot": torch.empty(case["nt"], dtype=torch.float64, device="cuda")}
    X, T, p = _mlp_data(case, seed)
    return {"kind": kind, "K": K, "shape": (case["F"], case["H"], case["O"]), "X": X, "T": T,
            "params": p, "steps": case["steps"]}


def run(state):
    K, kind = state["K"], state["kind"]
    stream = _handle()
    if kind == "solve":
        one = state["one"]
        one.set_sources(stream)
        one.plan.run(stream)
        return one.potentials(stream)
    if kind == "evaluate":
        f64 = ctypes.POINTER(ctypes.c_double)
        pts, pot = state["pts"], state["pot"]
        K.check(K.lib().kfmm_evaluate(state["plan"].handle,
                                      *[pts[k].ctypes.data_as(f64) for k in _SRC + _TRG],
                                      pot.ctypes.data_as(f64), stream), "evaluate")
        return pot
    if kind == "batch":
        for one in state["each"]:
            one.set_sources(stream)
        state["batch"].launch(stream)
        state["batch"].batch.wait(stream)
        return [one.potentials(stream) for one in state["each"]]
    if kind == "direct":
        pot = state["pot"].zero_()
        K.check(K.lib().kfmm_direct_evaluation(
            pot.numel(), *[t.data_ptr() for t in state["trg"]], pot.data_ptr(),
            state["src"][0].numel(), *[t.data_ptr() for t in state["src"]], stream), "direct")
        return pot
    net = K.MLP(*state["shape"], params=state["params"].copy())
    losses = net.train(state["X"], state["T"], state["steps"], 2e-3)
    return {"params": net.params, "losses": losses}


def _solve_flops(dist, n, ppb, np_):
    """Near-field pairs at 11 flops, V-list products at 8, S2M pairs and the
    level products at 2, on a full tree of boxes of the mean occupancy."""
    P = np_ ** 3 - (np_ - 2) ** 3
    Q = (np_ + 2) ** 3 - np_ ** 3
    F = (np_ + 1) * (2 * np_) ** 2
    grow, near, far = (8, 27, 189) if dist == "uniform" else (4, 9, 27)
    depth = max(0, math.ceil(math.log(max(1.0, n / ppb), grow)))
    boxes = grow ** depth
    return (11.0 * n * near * n / boxes + 11.0 * n * (Q + P) + 8.0 * boxes * far * F
            + 2.0 * boxes * (P * Q + 4 * P * P))


def work(case):
    kind = case["kind"]
    if kind in ("solve", "evaluate"):
        return {"bytes": 64.0 * case["n"],
                "flops": _solve_flops(case["dist"], case["n"], case["ppb"], case["np"])}
    if kind == "batch":
        _package()
        sp = _batch_specs(case, 0)
        return {"bytes": 64.0 * sum(s["n"] for s in sp),
                "flops": sum(_solve_flops(s["distribution"], s["n"], 64, s["np"]) for s in sp)}
    if kind == "direct":
        return {"bytes": 32.0 * (case["ns"] + case["nt"]), "flops": 11.0 * case["ns"] * case["nt"]}
    F, H, O, B = case["F"], case["H"], case["O"], case["B"]
    return {"bytes": 4.0 * B * (F + O),
            "flops": case["steps"] * 2.0 * B * (2 * F * H + 3 * H * H + 3 * H * O)}


# Plain FP64 form: the pseudo-inverses amplify a reordering of the sums by up to
# their condition number 0.1^-(np+1).  Split-K factors 1, 2 and 16 of the level
# products against the automatic ones moved the potentials by 1.4e-14, 2.7e-13,
# 2.6e-12, 2.0e-11, 1.5e-10 and 1.6e-9 at NP 3 to 8 (the largest of uniform,
# ellipse and ellipsoid-surface clouds of 20,000 to 1,048,576 points).
_FP64_REL = {3: 1e-13, 4: 1e-12, 5: 1e-11, 6: 8e-11, 7: 6e-10, 8: 6e-9}
# Mixed form: FP32 coordinates relative to the box and FP32 pair terms; its
# distance to the plain form was 8.9e-8 on uniform clouds, 2.3e-7 on the ellipse
# and 2.9e-5 on the ellipsoid surface (crowded poles, densities of both signs).
_MIXED_REL = {"uniform": 4e-7, "ellipseUniformAngles": 1e-6, "ellipsoidSurface": 1e-4}


def tolerance(case):
    kind = case["kind"]
    if kind in ("solve", "evaluate"):
        return {"rel": _FP64_REL[case["np"]] if case["prec"] == "fp64" else _MIXED_REL[case["dist"]]}
    if kind == "batch":  # NP 3 and 4, uniform and ellipsoid surface
        return {"rel": _FP64_REL[4] if case["prec"] == "fp64" else _MIXED_REL["ellipsoidSurface"]}
    if kind == "direct":  # up to 2.7e-14 from the sum in torch's order
        return {"rel": 1e-13}
    # FP32 sums over the batch, then Adam's normalised steps: parameters 6.6e-6
    # and losses 3.7e-6 from the same steps in FP64
    return {"rel": 3e-5, "max": 5e-3}


def _direct64(src, trg):
    """1/(4 pi) sum_j w_j / |t_i - s_j| over the sources away from the target."""
    sx, sy, sz, w = src
    tx, ty, tz = trg
    out = torch.empty_like(tx)
    step = max(1, (1 << 28) // sx.numel())
    for i in range(0, tx.numel(), step):
        s = slice(i, i + step)
        d = tx[s, None] - sx[None]
        r2 = d.mul_(d)
        for t, c in ((ty, sy), (tz, sz)):
            d = t[s, None] - c[None]
            r2.addcmul_(d, d)
        inv = r2.rsqrt_()
        inv.masked_fill_(torch.isinf(inv), 0.0)
        out[s] = inv @ w
    return out / (4.0 * math.pi)


def _exact_solve(dist, n, coincide, seed):
    pts = _package().generate_points(n, dist, coincide, seed)  # the inputs alone
    return _direct64([torch.from_numpy(pts[k]).cuda() for k in _SRC],
                     [torch.from_numpy(pts[k]).cuda() for k in _TRG])


def _exact_mlp(case, seed):
    X, T, p = _mlp_data(case, seed)
    F, H, O = case["F"], case["H"], case["O"]
    X, T, p = (torch.from_numpy(a).double().cuda() for a in (X, T, p))
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for s in range(1, case["steps"] + 1):
        p.requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = torch.split(p, [F * H, H, H * H, H, H * O, O])
        h = torch.relu(X @ w1.view(F, H) + b1)
        h = torch.relu(h @ w2.view(H, H) + b2)
        loss = ((h @ w3.view(H, O) + b3 - T) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        p = p.detach()
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 2e-3 * (m / (1 - 0.9 ** s)) / ((v / (1 - 0.999 ** s)).sqrt() + 1e-8)
    return {"params": p.cpu().numpy(), "losses": np.array(losses)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "evaluate"):
        # over 300,000 points the direct sum takes too long
        if case["n"] > 300000:
            return None
        out = _exact_solve(case["dist"], case["n"], case["coincide"], seed)
        return out.cpu().numpy() if kind == "evaluate" else out
    if kind == "batch":
        return [_exact_solve(s["distribution"], s["n"], 0, s["seed"])
                for s in _batch_specs(case, seed)]
    if kind == "direct":
        return _direct64(*_check_points(case, seed))
    return _exact_mlp(case, seed)
