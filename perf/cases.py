"""Performance cases: the calls a user of the tracker makes, through its public entry points.

Kinds of call (one case = one call, or one short sequence of calls a program makes per round):

  track    Tracker.track on Stephenson II tasks: host tasks in, host roots, codes and residuals out
  rounds   Tracker.track_rounds: several rounds in flight, host buffers, as the multi-round driver runs
  plugin   Tracker.track / track_into on a plug-in system (conic2, burmester5)
  collect  a DeviceCollection from empty: several rounds of roots merged one after another

A path is tracked step by step, every step waiting for the one before it, and paths differ
widely in length, so a call of up to some thousand paths takes as long as its longest path.
The sizes below span the test suite's calls (8 to 1,024 Stephenson II paths, 64 to
262,144 plug-in paths) and the collection's benchmark size (65,536 roots); the FP64 budget
of the larger mixed-precision calls bounds their longest path, as a program that wants an
answer within a second or so would.
"""
from __future__ import annotations

import numpy as np
import torch

import finite_root_generation_gb300 as frg
from finite_root_generation_gb300.systems import burmester5
from finite_root_generation_gb300.tasks import REFERENCE_TARGET, precision_point_task

# Algorithmic cost of one linear-system step (FLOP: complex mul 6, add 2) and the usual
# number of steps a path takes, per system.
FLOP_PER_SOLVE = {"stephenson2": 37930, "conic2": 1026, "burmester5": 3110}
SOLVES_PER_PATH = {"stephenson2": 1300, "conic2": 107, "burmester5": 290}
UNKNOWNS = {"stephenson2": 21, "conic2": 2, "burmester5": 5}
PARAMS = {"stephenson2": 30, "conic2": 12, "burmester5": 20}


def listed():
    return [
        # a first look at a task: a handful of paths in the reference's arithmetic and settings
        {"name": "track_fp64_8", "kind": "track", "precision": "fp64", "target": "reference", "ntasks": 1, "paths": 8},
        # two precision-point tasks of unequal path counts, endpoints asked for as well
        {"name": "track_fp64_ragged", "kind": "track", "precision": "fp64", "target": "points", "ntasks": 2,
         "paths": 9, "yfinal": True},
        # a whole FP64 round on the reference target, small enough that the GPU is not full
        {"name": "track_fp64_200", "kind": "track", "precision": "fp64", "target": "reference", "ntasks": 1,
         "paths": 200},
        # the benchmark's mixed-precision setting on few paths
        {"name": "track_mixed_13", "kind": "track", "precision": "mixed", "target": "points", "ntasks": 1,
         "paths": 13},
        # mixed precision on the reference target with the reference's uniform starts
        {"name": "track_mixed_150", "kind": "track", "precision": "mixed", "target": "reference", "ntasks": 1,
         "paths": 150, "budget": 3000},
        # a mixed round over several tasks that fills a good part of the GPU
        {"name": "track_mixed_2048", "kind": "track", "precision": "mixed", "target": "points", "ntasks": 4,
         "paths": 512, "budget": 2000},
        # four rounds in flight, paths carried between them (the multi-round driver's call)
        {"name": "rounds_mixed_4x300", "kind": "rounds", "target": "points", "rounds": 4, "depth": 4, "paths": 300,
         "budget": 2000},
        # the smallest system: one small round in mixed precision, launches and latency count
        {"name": "conic2_mixed_64", "kind": "plugin", "system": "conic2", "precision": "mixed", "ntasks": 1,
         "paths": 64},
        # the smallest system, a full GPU in FP64
        {"name": "conic2_fp64_262144", "kind": "plugin", "system": "conic2", "precision": "fp64", "ntasks": 64,
         "paths": 4096},
        # five-position Burmester dyads of one motion, FP64, odd count
        {"name": "burmester5_fp64_777", "kind": "plugin", "system": "burmester5", "precision": "fp64", "ntasks": 1,
         "paths": 777},
        # the same in mixed precision over several motions, device buffers
        {"name": "burmester5_mixed_3000", "kind": "plugin", "system": "burmester5", "precision": "mixed",
         "ntasks": 3, "paths": 1000, "device": True},
        # the collection of eight tasks over four rounds of 65,536 roots, some of them known already
        {"name": "collect_4x65536", "kind": "collect", "rounds": 4, "roots": 65536, "keys": 8},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["track", "track", "rounds", "plugin", "plugin", "plugin", "collect"])
    if kind == "track":
        prec = rng.choice(["fp64", "mixed"])
        target = rng.choice(["reference", "points"])
        c = {"kind": "track", "precision": prec, "target": target, "ntasks": rng.randint(1, 3)}
        if prec == "fp64":
            c["paths"] = _log(rng, 2, 64 if target == "reference" else 6)
            c["yfinal"] = rng.random() < 0.3
        else:
            c["paths"] = _log(rng, 2, 200)
            c["budget"] = rng.choice([1000, 2000])
        return c
    if kind == "rounds":
        r = rng.randint(2, 4)
        return {"kind": "rounds", "target": rng.choice(["reference", "points"]), "rounds": r, "depth": r,
                "paths": _log(rng, 8, 250), "budget": 1000}
    if kind == "plugin":
        system = rng.choice(["conic2", "burmester5"])
        prec = rng.choice(["fp64", "mixed"])
        hi = 4096 if system == "conic2" else 700
        return {"kind": "plugin", "system": system, "precision": prec, "ntasks": rng.randint(1, 9) if system == "conic2"
                else rng.randint(1, 3), "paths": _log(rng, 16, hi), "device": rng.random() < 0.5}
    return {"kind": "collect", "rounds": rng.randint(1, 5), "roots": _log(rng, 100, 65536), "keys": rng.randint(1, 16)}


def _targets(case, seed, n):
    """n Stephenson II tasks: the reference's target, or precision-point tasks (disk and curve in turn)."""
    if case["target"] == "reference":
        return np.repeat(REFERENCE_TARGET[None, :], n, axis=0)
    return np.stack([precision_point_task(1000 * seed + k, "disk" if k % 2 == 0 else "curve") for k in range(n)])


def _config(case):
    """The reference's settings on its own target; the benchmark's starts, gamma and finite-root
    test on precision-point tasks. Mixed precision is the chosen setting."""
    kw = {}
    if case["target"] == "points":
        kw = dict(start_dist=frg.START_NORMAL, gamma_mode=frg.GAMMA_RANDOM, inf_tol=1e-8)
    if case.get("budget"):
        kw["fp64_budget"] = case["budget"]
    mixed = case["kind"] == "rounds" or case["precision"] == "mixed"
    return frg.chosen_config(**kw) if mixed else frg.default_config(**kw)


def _counts(case):
    """Paths per task: the case's count, one fewer for every further task (ragged offsets)."""
    return [max(1, case["paths"] - k) for k in range(case["ntasks"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": int(seed)}
    if kind == "track":
        s["tasks"], s["ppt"] = _targets(case, seed, case["ntasks"]), _counts(case)
        s["tracker"] = frg.Tracker(_config(case))
    elif kind == "rounds":
        r, n = case["rounds"], case["paths"]
        s["tasks"] = _targets(case, seed, 1)
        s["seeds"] = [seed * 100 + k for k in range(r)]
        s["roots"], s["codes"] = np.zeros((r * n, 21), np.complex128), np.zeros(r * n, np.int32)
        s["resid"] = np.zeros(r * n, np.float64)
        s["tracker"] = frg.Tracker(_config(case))
    elif kind == "plugin":
        rng = np.random.default_rng(seed)
        nt = case["ntasks"]
        if case["system"] == "conic2":
            s["tasks"] = rng.normal(size=(nt, 12)) + 1j * rng.normal(size=(nt, 12))
        else:
            s["tasks"] = np.stack([burmester5.physical_task(rng) for _ in range(nt)])
        s["ppt"] = [case["paths"]] * nt
        prec = frg.PREC_MIXED if case["precision"] == "mixed" else frg.PREC_FP64
        cfg = frg.plugin_config(case["system"], precision=prec, start_dist=frg.START_NORMAL,
                                gamma_mode=frg.GAMMA_RANDOM, inf_tol=1e-8)
        s["tracker"] = frg.Tracker(cfg)
        if case.get("device"):
            n, nv = sum(s["ppt"]), UNKNOWNS[case["system"]]
            s["fpm"] = torch.from_numpy(np.ascontiguousarray(s["tasks"]).view(np.float64)).cuda()
            s["roots"] = torch.zeros((n, 2 * nv), dtype=torch.float64, device="cuda")
            s["codes"] = torch.zeros(n, dtype=torch.int32, device="cuda")
            s["resid"] = torch.zeros(n, dtype=torch.float64, device="cuda")
    else:
        # rounds of roots as tracking leaves them: a few per cent failed paths, and in each
        # round some roots of the rounds before it found again to about 1e-13
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        n = case["roots"]
        s["sets"], prev = [], None
        for _ in range(case["rounds"]):
            roots = 3.0 * torch.randn((n, 42), dtype=torch.float64, device="cuda", generator=g)
            keys = torch.randint(0, case["keys"], (n,), dtype=torch.int32, device="cuda", generator=g)
            codes = torch.where(torch.rand(n, device="cuda", generator=g) < 0.98, 0, 2).to(torch.int32)
            if prev is not None:
                m = n // 5
                pick = torch.randint(0, n, (m,), device="cuda", generator=g)
                noise = 1e-13 * torch.randn((m, 42), dtype=torch.float64, device="cuda", generator=g)
                roots[:m], keys[:m] = prev[0][pick] + noise, prev[1][pick]
            resid = 1e-14 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
            s["sets"].append((roots, codes, keys, resid))
            prev = (roots, keys)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "track":
        r = state["tracker"].track(state["tasks"], state["ppt"], state["seed"], want_yfinal=bool(case.get("yfinal")),
                                   want_resid=True)
        return {"roots": r.roots, "codes": r.codes, "yfinal": r.yfinal, "resid": r.resid}
    if kind == "rounds":
        state["tracker"].track_rounds(state["tasks"], [case["paths"]], state["seeds"], state["roots"], state["codes"],
                                      resid=state["resid"], depth=case["depth"])
        return {"roots": state["roots"], "codes": state["codes"], "resid": state["resid"]}
    if kind == "plugin":
        if case.get("device"):
            state["tracker"].track_into(state["fpm"], state["ppt"], state["seed"], state["roots"], state["codes"],
                                        resid=state["resid"])
            return {"roots": state["roots"], "codes": state["codes"], "resid": state["resid"]}
        r = state["tracker"].track(state["tasks"], state["ppt"], state["seed"], want_resid=True)
        return {"roots": r.roots, "codes": r.codes, "resid": r.resid}
    coll = frg.DeviceCollection(case["rounds"] * case["roots"])
    marked = []
    for roots, codes, keys, resid in state["sets"]:
        c = codes.clone()
        coll.merge(roots, c, keys, stream=torch.cuda.current_stream().cuda_stream, resid=resid)
        marked.append(c)
    size = coll.size(torch.cuda.current_stream().cuda_stream)
    coll.close()
    return {"codes": marked, "size": size}


def work(case):
    """Bytes: tasks and start draws read once, roots, codes and residuals written once
    (collection: the rounds' roots, codes, keys and residuals read, new roots and codes
    written). FLOP: the linear-system steps the paths need."""
    if case["kind"] == "collect":
        n = case["rounds"] * case["roots"]
        return {"bytes": n * (2 * 42 * 8 + 2 * 4 + 4 + 8), "flops": 0}
    system = case.get("system", "stephenson2")
    nv, np_ = UNKNOWNS[system], PARAMS[system]
    n = case["rounds"] * case["paths"] if case["kind"] == "rounds" else (
        sum(_counts(case)) if case["kind"] == "track" else case["ntasks"] * case["paths"])
    per = 16 * nv + 4 + 8 + (16 * (nv + 2) if case.get("yfinal") else 0)
    return {"bytes": n * per + 16 * np_ * case.get("ntasks", 1),
            "flops": n * SOLVES_PER_PATH[system] * FLOP_PER_SOLVE[system]}


def exact(case, seed):
    """None: which root a path reaches is decided by some thousand dependent adaptive steps of
    this tracker on its own random streams, and the collection's outputs are whole numbers."""
    return None
