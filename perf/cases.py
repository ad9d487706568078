"""Performance cases: the work a user of this framework has it do, through its public entry points.

Every case is one call sequence of a search program: score a population of programs against a
dataset (`secant_cubin_runner_run`, host programs every call), the same against device-resident
programs, predictions and statistics of static programs, and rollout scoring of candidate ODE
right-hand sides (`secant_b200_rk4_score`, `odezza_scoring_pipeline_run`), with the reductions that
follow.  Populations and data are seeded synthetic stand-ins in the shapes of this repository's
benchmark configurations and tests.

A case is a dict of plain values; `prepare` makes its inputs on the GPU from a seed, `run` is one
pass, `work` counts what a pass cannot do without, `tolerance` what two correct implementations
of the same precision may differ by.
"""
import ctypes as C
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-program-specialization_b200"))

from secant_b200 import abi, engine as E, programs as P  # noqa: E402
from secant_b200.runner import (Runner, best_config, grouped_topk, rk4_score, score_fields, topk)  # noqa: E402

# ------------------------------------------------------------------------------- cases ----


def _static(shape, programs, tokens, rows, features, targets=1):
    return dict(kind="static", shape=shape, programs=programs, tokens=tokens, rows=rows, features=features, targets=targets)


def _scoring(programs, tokens, rows, features, slots, sets, bits, gated=False, own_banks=False, fast=False, resident=False, top=0):
    return dict(kind="scoring", programs=programs, tokens=tokens, rows=rows, features=features, slots=slots, sets=sets, bits=bits,
                gated=gated, own_banks=own_banks, fast=fast, resident=resident, top=top)


def _rollout(systems, states, tokens, slots, trajectories, steps):
    return dict(kind="rollout", systems=systems, states=states, tokens=tokens, slots=slots, trajectories=trajectories, steps=steps)


def _engine(systems, states, tokens, slots, sets, bits, trajectories, points, substeps, top):
    return dict(kind="engine", systems=systems, states=states, tokens=tokens, slots=slots, sets=sets, bits=bits, trajectories=trajectories,
                points=points, substeps=substeps, top=top)


def listed():
    return [
        # the smallest scoring call: the CPU-checkable configuration (64 short programs, 4,096 rows)
        dict(_static("sse", 64, 15, 4096, 4), name="static_sse_small"),
        # a toggle search on a handful of rows: 129 programs x 5 sets x 256 variants, and the winners
        dict(_scoring(129, 24, 97, 4, 4, 5, 8, top=16), name="toggles_few_rows"),
        # one generation of a symbolic-regression search: every toggle variant of 1,000 programs on an
        # ordinary table of measurements, the best variant of each, the best programs of all
        dict(_scoring(1000, 32, 2001, 5, 8, 1, 8, top=100), name="search_generation"),
        # a population against 64 coefficient sets of its own, fused squared error: the headline shape
        dict(_scoring(2048, 32, 131072, 8, 16, 64, 0, own_banks=True, top=1024), name="population_64_sets"),
        # first screening on a wide, long dataset with the approximate functions, 16 shared sets
        dict(_scoring(1024, 32, 1048583, 16, 16, 16, 0, fast=True), name="wide_screening_fast"),
        # subtrees gated by toggles: 256 variants x 4 sets of each program, and its best variant
        dict(_scoring(384, 48, 32768, 6, 8, 4, 8, gated=True, top=64), name="gated_subtrees"),
        # refinement of the survivors: resident programs scored again with new coefficient sets
        dict(_scoring(256, 32, 10007, 6, 12, 33, 0, resident=True), name="resident_refinement"),
        # predictions of a population for every row
        dict(_static("materialize", 500, 24, 100003, 6, 0), name="predictions"),
        # affine-fit statistics (sums, squares, cross sums with two targets) of a feature pool
        dict(_static("affine", 3000, 24, 20011, 6, 2), name="affine_statistics"),
        # cohort Gram matrices of candidate features (8 per cohort) for a sparse-regression solver
        dict(_static("gram", 512, 15, 65536, 5, 2), name="gram_statistics"),
        # candidate right-hand sides of a 3-state system against 64 reference trajectories
        dict(_rollout(4096, 3, 24, 8, 64, 1000), name="rollout_uniform"),
        # the ODE engine's launch: ragged trajectories with missing observations, several coefficient
        # sets, toggles; then the best configurations of every system
        dict(_engine(600, 2, 14, 3, 3, 2, 37, 24, 2, 16), name="rollout_engine"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One more case of the same ranges: sizes log-uniform, mostly odd, its cost within the listed ones'."""
    kind = rng.choice(["sse", "materialize", "affine", "gram", "toggles", "sets", "sets", "gated", "resident", "rollout", "engine"])
    tokens = rng.randint(10, 32)
    if kind in ("sse", "materialize", "affine", "gram"):
        programs = _log_int(rng, 50, 4000)
        most = {"sse": 1e8, "materialize": 5e7, "affine": 6e7, "gram": 3.3e7}[kind]
        rows = _log_int(rng, 1000, max(1001, min(400000, int(most / programs))))
        targets = 0 if kind == "materialize" else 1 if kind == "sse" else rng.randint(1, 3)
        return _static(kind, programs, min(tokens, 24), rows, rng.randint(3, 12), targets)
    if kind == "toggles":
        bits, sets, programs = rng.randint(4, 9), rng.choice([1, 1, 2, 5]), _log_int(rng, 60, 2000)
        most = max(65, min(20000, int(6e8 / (programs * (sets << bits)))))
        return _scoring(programs, tokens, _log_int(rng, 64, most), rng.randint(2, 8), rng.randint(4, 12), sets, bits, top=rng.choice([0, 16, 50]))
    if kind in ("sets", "resident"):
        resident = kind == "resident"
        sets = rng.choice([1, 3, 8, 16, 20, 33, 64])
        programs = _log_int(rng, 100, 1000 if resident else 4000)
        most = max(1001, min(1200000, int((2e9 if resident else 1.5e10) / (programs * sets))))
        return _scoring(programs, tokens, _log_int(rng, 1000, most), rng.randint(3, 16), rng.randint(4, 16), sets, 0,
                        own_banks=rng.random() < 0.5, fast=rng.random() < 0.25, resident=resident, top=0 if resident else rng.choice([0, 20]))
    if kind == "gated":
        bits, sets, programs = rng.randint(5, 8), rng.choice([1, 2, 4, 6]), _log_int(rng, 50, 600)
        most = max(1001, min(100000, int(1e10 / (programs * (sets << bits)))))
        return _scoring(programs, rng.randint(30, 48), _log_int(rng, 1000, most), rng.randint(3, 8), rng.randint(4, 12), sets, bits, gated=True, top=20)
    if kind == "rollout":
        systems, trajectories = _log_int(rng, 200, 4000), rng.choice([16, 20, 32, 50, 64, 130])
        most = max(51, min(1500, int(2.5e8 / (systems * trajectories))))
        return _rollout(systems, rng.randint(1, 4), min(tokens, 24), rng.randint(2, 10), trajectories, _log_int(rng, 50, most))
    return _engine(_log_int(rng, 100, 900), rng.randint(1, 3), rng.randint(8, 20), rng.randint(2, 6), rng.choice([1, 2, 3]), rng.choice([0, 1, 2]),
                   rng.randint(5, 40), rng.randint(8, 40), rng.randint(1, 4), rng.choice([4, 16, 32]))


# ----------------------------------------------------------------------------- inputs ----

_TAME = [(P.op("ADD"), 2), (P.op("SUB"), 2), (P.op("MUL"), 2), (P.op("SIN"), 1), (P.op("COS"), 1), (P.op("TANH"), 1)]
_SHAPES = {"sse": abi.SHAPE_SSE, "materialize": abi.SHAPE_MATERIALIZE, "affine": abi.SHAPE_AFFINE_STATS, "gram": abi.SHAPE_GRAM_STATS}
_COHORT = 8
_DT = 0.01
_handles = {}  # a search program keeps one runner (or pipeline) per kind of call for as long as it lives


def _runner(shape, features, targets, slots, fast=False):
    key = (shape, features, targets, slots, fast)
    if key not in _handles:
        rn = Runner(shape, features, targets, slots, workers=4, streams=2, asts_per_kernel=_COHORT if shape == abi.SHAPE_GRAM_STATS else None)
        rn.set_math(fast)
        _handles[key] = rn
    return _handles[key]


def _pipeline(states, slots):
    key = ("engine", states, slots)
    if key not in _handles:
        _handles[key] = E.ScoringPipeline(states, slots)
    return _handles[key]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _table(g, features, targets, rows, spread, gaussian=False):
    """Measurements: [feature][row] and noisy targets of a hidden expression, [target][row]."""
    if gaussian:
        x = torch.randn((features, rows), generator=g, device="cuda")
    else:
        x = (torch.rand((features, rows), generator=g, device="cuda") * 2 - 1) * spread
    noise = 0.05 * torch.randn((max(1, targets), rows), generator=g, device="cuda")
    hidden = x[0] * x[1] + torch.sin(x[min(2, features - 1)])
    return x, hidden[None, :] + noise


def _prepare_static(c, seed):
    g = _generator(seed)
    gram = c["shape"] == "gram"
    pop = P.random_population(seed, c["programs"], c["tokens"], c["features"], 0, 1.0, ops=_TAME if gram else None)
    x, y = _table(g, c["features"], c["targets"], c["rows"], 1.0)
    rn = _runner(_SHAPES[c["shape"]], c["features"], max(1, c["targets"]), 0)
    if c["shape"] == "materialize":
        out = torch.zeros((c["programs"], c["rows"]), device="cuda")
        request = rn.materialize_request(pop, x, out)
    else:
        if gram:
            shape = ((c["programs"] + _COHORT - 1) // _COHORT, _COHORT * (1 + _COHORT + c["targets"]))
        else:
            shape = (c["programs"], c["targets"] + (2 if c["shape"] == "affine" else 0))
        out = torch.zeros(shape, device="cuda")
        request = rn.static_request(pop, x, y, out)
    return dict(call=rn.run, request=request, out=out, top=0, keep=(pop, x, y))


def _prepare_scoring(c, seed):
    g = _generator(seed)
    programs, slots, sets = c["programs"], c["slots"], c["sets"]
    if c["gated"]:
        pop = P.gated_population(seed, programs, c["tokens"], c["features"], slots, c["bits"])
    else:
        pop = P.random_population(seed, programs, c["tokens"], c["features"], slots, 3.0, toggle_bits=c["bits"])
    x, y = _table(g, c["features"], 1, c["rows"], 3.0, gaussian=c["gated"])
    tables = programs if c["own_banks"] else 1
    banks = torch.randn((tables, sets, slots), generator=g, device="cuda")
    out = torch.zeros((programs, 1, sets << c["bits"]), device="cuda")
    rn = _runner(abi.SHAPE_TOGGLE_SSE, c["features"], 1, slots, c["fast"])
    request = rn.toggle_request(pop, x, y, banks, sets, c["bits"], out, bank_stride=slots,
                                program_bank_stride=sets * slots if c["own_banks"] else 0)
    call = rn.run
    if c["resident"]:
        call = _Resident(rn, pop, c["bits"]).run
    return dict(call=call, request=request, out=out, top=min(c["top"], programs), keep=(pop, x, y, banks))


class _Resident:
    """A resident population given back when its state goes."""

    def __init__(self, rn, pop, bits):
        self.population = rn.population(pop, bits)
        self.run = self._run

    def _run(self, request):
        return self.population.run(request)

    def __del__(self):
        self.population.destroy()


def _lorenz(rng, trajectories, points):
    """[3][trajectory][point] of the Lorenz system from seeded initial conditions."""
    h = np.float32(_DT)
    v = rng.uniform(-10, 10, size=(3, trajectories)).astype(np.float32)
    out = np.empty((3, trajectories, points), dtype=np.float32)
    out[:, :, 0] = v

    def rhs(s):
        return np.stack([(s[1] - s[0]) * np.float32(10), s[0] * (np.float32(28) - s[2]) - s[1], s[0] * s[1] - np.float32(8 / 3) * s[2]])

    for k in range(1, points):
        k1 = rhs(v)
        k2 = rhs(v + h / 2 * k1)
        k3 = rhs(v + h / 2 * k2)
        k4 = rhs(v + h * k3)
        v = (v + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)).astype(np.float32)
        out[:, :, k] = v
    return out


def _prepare_rollout(c, seed):
    rng = np.random.default_rng(seed)
    states, points = c["states"], c["steps"] + 1
    pop = P.random_population(seed, c["systems"] * states, c["tokens"], states, c["slots"], 1.0)
    paths = _lorenz(rng, c["trajectories"], points)
    paths = np.concatenate([paths, paths[:1] * np.float32(0.5)])[:states]
    reference = torch.from_numpy(np.ascontiguousarray(paths.reshape(states, -1))).cuda()
    times = torch.from_numpy(np.arange(points, dtype=np.float32) * np.float32(_DT)).cuda()
    coefficients = torch.randn((c["systems"], 1, c["slots"]), generator=_generator(seed), device="cuda")
    return dict(pop=pop, reference=reference, times=times, coefficients=coefficients, states=states, slots=c["slots"])


_ENGINE_TOKEN = {"RET": "RET", "COL": "STATE", "BANK": "CONSTANT"}


def _engine_bytes(code):
    """A postfix program in the ODE engine's token values (operand bytes unchanged)."""
    names = {v: k for k, v in P.OP.items()}
    wide = {"COL": 2, "BANK": 2, "LIT": 5, "TOG2": 2, "TOG4": 3}
    out, at = bytearray(), 0
    while at < len(code):
        name = names[code[at]]
        width = wide.get(name, 1)
        out.append(E.OP[_ENGINE_TOKEN.get(name, name)])
        out += code[at + 1:at + width]
        at += width
    return bytes(out)


def _prepare_engine(c, seed):
    rng = np.random.default_rng(seed)
    states, systems, configs = c["states"], c["systems"], c["sets"] << c["bits"]
    raw = P.random_population(seed, systems * states, c["tokens"], states, c["slots"], 1.0, toggle_bits=c["bits"], ops=_TAME)
    # contracting right-hand sides, as a candidate of a search that is under way: tanh(f) - x
    sides = [_engine_bytes(a[:-1] + P.op("TANH") + P.col(i % states) + P.op("SUB") + P.RET) for i, a in enumerate(raw.asts)]
    array, keep = E.systems_array([[(s, sides[i * states + s]) for s in range(states)] for i in range(systems)])
    lengths = rng.integers(2, c["points"] + 1, size=c["trajectories"])
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    times = np.concatenate([np.cumsum(rng.uniform(0.02, 0.07, size=n)) for n in lengths]).astype(np.float32)
    reference = rng.uniform(-1, 1, size=(states, int(offsets[-1]))).astype(np.float32)
    holes = rng.random(reference.shape) < 0.05
    holes[:, offsets[:-1]] = False  # a first point is an initial condition
    reference[holes] = np.nan
    dev = dict(offsets=torch.from_numpy(offsets).cuda(), times=torch.from_numpy(times).cuda(), reference=torch.from_numpy(reference).cuda(),
               banks=torch.randn((systems, c["sets"], c["slots"]), generator=_generator(seed), device="cuda"),
               out=torch.zeros((systems, configs), device="cuda"))
    launch = E.Launch()
    launch.constant_banks_device = dev["banks"].data_ptr()
    launch.constant_bank_count, launch.active_toggle_count = c["sets"], c["bits"]
    launch.trajectory_offsets_device, launch.trajectory_times_device = dev["offsets"].data_ptr(), dev["times"].data_ptr()
    launch.reference_data_device, launch.mse_output_device = dev["reference"].data_ptr(), dev["out"].data_ptr()
    launch.trajectory_count, launch.trajectory_point_count = c["trajectories"], int(offsets[-1])
    launch.steps_per_observation = c["substeps"]
    launch.allow_missing_observations = 1
    return dict(pipe=_pipeline(states, c["slots"]), array=array, launch=launch, report=E.RunReport(), case=c, keep=(keep, dev), out=dev["out"])


def prepare(case, seed):
    make = {"static": _prepare_static, "scoring": _prepare_scoring, "rollout": _prepare_rollout, "engine": _prepare_engine}
    state = make[case["kind"]](case, seed)
    torch.cuda.synchronize()  # the library does not wait for work queued on the caller's streams
    return dict(state, kind=case["kind"])


# ------------------------------------------------------------------------------- a pass ----


def run(state):
    if state["kind"] == "rollout":
        return rk4_score(state["pop"], state["states"], state["reference"], state["times"], state["coefficients"], state["slots"])
    if state["kind"] == "engine":
        c, pipe = state["case"], state["pipe"]
        E.check(pipe.lib.odezza_scoring_pipeline_run(pipe.handle, state["array"], c["systems"], C.byref(state["launch"]), pipe.workspace,
                                                     pipe.workspace_size, C.byref(state["report"])), "odezza_scoring_pipeline_run")
        k = min(c["top"], c["sets"] << c["bits"])
        mse, index, counts = grouped_topk(state["out"], c["systems"], c["sets"], c["bits"], E.BY_SYSTEM, k)
        torch.cuda.current_stream().synchronize()  # the search reads the winners before it goes on
        return dict(scores=state["out"], mse=mse, index=index, counts=counts)
    state["call"](state["request"])
    if not state["top"]:
        return state["out"]
    best = best_config(state["out"])
    sse, configuration, valid = score_fields(best)
    programs, values = topk(sse, state["top"])
    torch.cuda.current_stream().synchronize()  # the search reads the winners before it makes the next generation
    return dict(scores=state["out"], best=sse, configuration=configuration, valid=valid, programs=programs, values=values)


def work(case):
    c = case
    operations = 0.6 * c["tokens"]  # arithmetic nodes of a random program of at most `tokens` tokens, routines inlined
    if c["kind"] == "static":
        cells = c["programs"] * c["rows"]
        data = 4 * c["rows"] * (c["features"] + c["targets"])
        if c["shape"] == "materialize":
            return {"bytes": data + 4 * cells, "flops": cells * operations}
        per = {"sse": 2 * c["targets"], "affine": 3 + 2 * c["targets"], "gram": 1 + _COHORT + 1 + 2 * c["targets"]}[c["shape"]]
        width = {"sse": c["targets"], "affine": 2 + c["targets"], "gram": 1 + _COHORT + c["targets"]}[c["shape"]]
        return {"bytes": data + 4 * c["programs"] * width, "flops": cells * (operations + per)}
    if c["kind"] == "scoring":
        configs = c["sets"] << c["bits"]
        tables = c["programs"] if c["own_banks"] else 1
        if c["bits"]:
            operations *= 0.6  # a toggled leaf is three tokens
        return {"bytes": 4 * (c["rows"] * (c["features"] + 1) + tables * c["sets"] * c["slots"] + c["programs"] * configs),
                "flops": c["programs"] * configs * c["rows"] * (operations + 2)}
    if c["kind"] == "rollout":
        evaluations = c["systems"] * c["states"] * c["trajectories"] * c["steps"] * 4
        return {"bytes": 4 * (c["states"] * c["trajectories"] * (c["steps"] + 1) + c["systems"] * (c["slots"] + 1)),
                "flops": evaluations * (operations + 4)}
    configs = c["sets"] << c["bits"]
    steps = c["trajectories"] * (c["points"] / 2) * c["substeps"]
    return {"bytes": 4 * (c["trajectories"] * c["points"] / 2 * (c["states"] + 1) + c["systems"] * configs * 2),
            "flops": c["systems"] * configs * c["states"] * steps * 4 * (operations + 4)}


def tolerance(case):
    """Sums of float32 products in another order, and functions within an ulp or two of each other under a few levels of
    exponentials: the losses of this repository are held to 1e-4 relative.  Near ties may swap two winners."""
    if case["kind"] == "static":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 1e-4, "max": 4e-3, "differ": 0.005}
