"""The grader's work as its users call it: cases to time and to compare.

A case names a shape (circuit sizes, pairs, table, options); prepare() makes
the netlists from the seed with the repository's generator and uniform random
pairs, and the circuit, state and batch handles that a program keeps;
run() is one pass through the public calls.  Circuits have the proportions of
the repository's workloads: primary inputs and outputs about a thirteenth of
the gates, fan-in 1 to 4, geometric fan-out unless the case says Zipf.
`types` is "all" (AND..XNOR, NOT, BUFF: the generator's default, where the
reference's tables send every multi-input XOR and XNOR to a constant) or
"plain" (without XOR and XNOR: no gate is constant).
"""
import ctypes
import importlib.util
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The package (its folder's name is no identifier)."""
    if "pdf_b200" not in sys.modules:
        path = os.path.join(_ROOT, "gpu-path-delay-coverage_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location("pdf_b200", path)
        mod = importlib.util.module_from_spec(spec)
        sys.modules["pdf_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["pdf_b200"]


P = _package()
PLAIN = sum(1 << t for t in (P.AND, P.NAND, P.OR, P.NOR, P.NOT, P.BUFF))
MODES = {"default": P.MARK_DEFAULT, "robust": P.MARK_ROBUST, "fixed_robust": P.MARK_FIXED_ROBUST,
         "fixed_nonrobust": P.MARK_FIXED_NONROBUST}


def listed():
    return [
        # the reference's smallest use: a 2,000-gate circuit, one chunk of 1,024 pairs, the count
        # waited for (fcount's default table)
        dict(name="small", kind="grade", gates=2000, pio=36, depth=40, types="all", pairs=1024, mode="default",
             chunks=1, host=False, planes=False, seg=1),
        # the plain single-circuit call at its usual size, --robust
        dict(name="medium", kind="grade", gates=20000, pio=1500, depth=60, types="all", pairs=32768, mode="robust",
             chunks=1, host=False, planes=False, seg=1),
        # fcount's chunk loop: host vectors of an odd count, graded in four chunks into one state, on a
        # circuit of gates that all switch
        dict(name="chunk_loop", kind="grade", gates=12001, pio=613, depth=45, types="plain", pairs=15001,
             mode="default", chunks=4, host=True, planes=False, seg=1),
        # every transition code and mark asked for (the --sim / --mark dumps, or a consumer on the device)
        dict(name="planes", kind="grade", gates=20000, pio=1500, depth=60, types="all", pairs=32768, mode="default",
             chunks=1, host=False, planes=True, seg=1),
        # the same on wide levels of gates that all switch
        dict(name="planes_wide", kind="grade", gates=150000, pio=8192, depth=40, types="plain", pairs=32768,
             mode="robust", chunks=1, host=False, planes=True, seg=1),
        # the largest circuit, Zipf fan-out, in a chunk that leaves room for its planes three times over
        dict(name="million", kind="grade", gates=1000000, pio=8192, depth=200, types="all", pairs=65536,
             mode="robust", chunks=1, host=False, planes=False, seg=1),
        # a large circuit of gates that all switch
        dict(name="large_plain", kind="grade", gates=200000, pio=15000, depth=80, types="plain", pairs=65536,
             mode="robust", chunks=1, host=False, planes=False, seg=1),
        # true n-input gates with the textbook robust table: marks reach many nets, counting weighs
        dict(name="fixed", kind="grade", gates=20000, pio=1500, depth=60, types="all", pairs=8192,
             mode="fixed_robust", chunks=1, host=False, planes=False, seg=1),
        # --segs 4
        dict(name="segments", kind="grade", gates=20000, pio=1500, depth=60, types="all", pairs=16384, mode="robust",
             chunks=1, host=False, planes=False, seg=4),
        # the reference's four host functions one after another over device planes
        dict(name="stages", kind="stages", gates=20000, pio=1500, depth=60, types="plain", pairs=16384,
             mode="default"),
        # many circuits of mixed sizes per pass, at the tile that the autotuner takes for such a batch
        dict(name="batch", kind="batch", jobs=40, gates_min=500, gates_max=200000, pairs_min=1024, pairs_max=65536,
             types="all", mode="robust", tile=128),
        # jobs that append: each pass grades the next 4,096 pairs of every job that has some left into the
        # states that its earlier passes left on the device, the batch bound anew for each pass at the
        # server's tile, as the serving loop does it (its host threads would be most of a timing)
        dict(name="append", kind="append", jobs=12, gates_min=2000, gates_max=100000, pairs_min=8192,
             pairs_max=65536, step=4096, types="all", mode="robust", tile=4),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choices(["grade", "stages", "batch", "append"], [6, 1, 2, 1])[0]
    types = rng.choice(["all", "plain"])
    mode = rng.choice(["default", "robust"])
    if kind == "batch":
        top = _log(rng, 2000, 100000)
        return dict(kind=kind, jobs=_log(rng, 4, 40), gates_min=500, gates_max=top, pairs_min=1024,
                    pairs_max=_log(rng, 2048, 32768), types=types, mode=mode, tile=rng.choice([0, 4, 8, 32, 64, 128]))
    if kind == "append":
        return dict(kind=kind, jobs=_log(rng, 4, 12), gates_min=2000, gates_max=_log(rng, 4000, 100000),
                    pairs_min=4096, pairs_max=_log(rng, 8192, 65536), step=rng.choice([1024, 2048, 4096, 8192]),
                    types=types, mode=mode, tile=rng.choice([4, 4, 8]))
    gates, pairs = _log(rng, 500, 200000), _log(rng, 32, 65536)
    pairs = max(32, min(pairs, 6_000_000_000 // gates))
    depth = min(rng.randint(10, 120), gates // 8)
    case = dict(kind=kind, gates=gates, pio=max(16, gates // rng.randint(8, 40)), depth=depth, types=types,
                pairs=pairs, mode=mode)
    if kind == "grade":
        case.update(chunks=rng.choice([1, 1, 1, 2, 3]), host=rng.random() < 0.25, planes=False, seg=1)
        option = rng.choice(["none", "none", "planes", "fixed", "segments"])
        if option == "planes":
            case.update(planes=True, host=False, chunks=1)
        elif option == "fixed":
            case.update(mode=rng.choice(["fixed_robust", "fixed_nonrobust"]), gates=max(500, gates // 8),
                        pairs=max(32, min(4096, pairs)))
            case.update(pio=max(16, case["gates"] // 13), depth=min(depth, case["gates"] // 8))
        elif option == "segments":
            case.update(seg=rng.randint(2, 4), gates=min(gates, 20000), pairs=min(pairs, 16384))
            case.update(pio=max(16, case["gates"] // 13), depth=min(depth, case["gates"] // 8))
    return case


def _netlist(case, seed):
    zipf = case["gates"] >= 500000
    return P.gen_netlist(P.GenParams(seed, case["gates"], case["pio"], min(case["pio"], case["gates"] - case["pio"]),
                                     case["depth"], fanout_dist=1 if zipf else 0, fanout_max=256 if zipf else 0,
                                     type_mask=PLAIN if case["types"] == "plain" else 0))


def _members(case):
    """(gates, depth, pairs) of each job of a batch: log-uniform sizes that belong to
    the case, not to the seed, so that every seed is the same amount of work."""
    rng = random.Random("%(jobs)d %(gates_min)d %(gates_max)d %(pairs_min)d %(pairs_max)d" % case)
    out = []
    for _ in range(case["jobs"]):
        gates = _log(rng, case["gates_min"], case["gates_max"])
        depth = rng.randint(20, 150)
        gates = max(gates, depth * 4)
        out.append((gates, depth, _log(rng, case["pairs_min"], case["pairs_max"])))
    return out


def _job_netlist(case, seed, k, gates, depth):
    pio = max(16, gates // 13)
    return _netlist(dict(gates=gates, pio=pio, depth=depth, types=case["types"]), seed * 1000 + k)


def _planes(gen, rows, words):
    return torch.randint(-2**31, 2**31, (rows, words), dtype=torch.int32, device="cuda", generator=gen)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed + 77)


def prepare(case, seed):
    seed = int(seed) % (1 << 40) + 1
    gen, mode = _generator(seed), MODES[case["mode"]]
    state = {"kind": case["kind"], "case": case}
    if case["kind"] in ("grade", "stages"):
        # the number of segments is the netlist's own, so there the netlist belongs to the case
        nl, n = _netlist(case, seed if case.get("seg", 1) == 1 else case["gates"]), case["pairs"]
        chunks = case.get("chunks", 1)
        step = -(-n // chunks)
        step = min(n, -(-step // 32) * 32)
        c = P.Circuit(nl, mark_mode=mode, max_pairs=step, seg_len=case.get("seg", 1))
        s = P.State(c)
        first = torch.empty((2, c.n_first), dtype=torch.int32, device="cuda")
        parts = []
        for base in range(0, n, step):
            m = min(step, n - base)
            v, t = _planes(gen, nl.n_pi, P.words(m)), _planes(gen, nl.n_pi, P.words(m))
            if case.get("host"):
                v, t = v.cpu().numpy().view(np.uint32), t.cpu().numpy().view(np.uint32)
            parts.append((base, m, v, t))
        out = None
        if case.get("planes") or case["kind"] == "stages":
            out = torch.empty((3, nl.n_gates, P.words(n)), dtype=torch.int32, device="cuda")
        state.update(c=c, s=s, first=first, parts=parts, out=out)
        return state
    step = case.get("step", 0)
    jobs, passes = [], []
    for k, (gates, depth, n) in enumerate(_members(case)):
        nl = _job_netlist(case, seed, k, gates, depth)
        c = P.Circuit(nl, mark_mode=mode, max_pairs=step or n, tile_words=case["tile"])
        s, tile = P.State(c), c.info().tile_words
        for i, base in enumerate(range(0, n, step or n)):
            m = min(step or n, n - base)
            ld = -(-P.words(m) // tile) * tile
            if i == len(passes):
                passes.append([])
            passes[i].append((c, s, _planes(gen, nl.n_pi, ld), _planes(gen, nl.n_pi, ld), m, base))
    jobs = passes[0]
    ends = np.cumsum([0] + [j[0].n_first for j in jobs])
    first = torch.empty((2, int(ends[-1])), dtype=torch.int32, device="cuda")
    state.update(jobs=jobs, passes=passes, batch=P.Batch(jobs, graph=not step), first=first,
                 views=[(first[0, a:b], first[1, a:b]) for a, b in zip(ends[:-1], ends[1:])])
    return state


def _halves(tot):
    """A 128-bit count as two 64-bit halves, and its flags."""
    return [tot.lo, tot.hi, tot.flags]


def run(state):
    kind = state["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "grade":
        c, s, out, counts = state["c"], state["s"], state["out"], []
        s.reset_async(stream)
        for base, m, v, t in state["parts"]:
            planes = dict(sim_v=out[0], sim_t=out[1], mark=out[2]) if out is not None else {}
            counts.append(_halves(P.grade(c, s, v, t, m, base, stream=stream, **planes)))
        P.first_copy(s, state["first"][0], state["first"][1], False, stream)
        result = {"count": np.array(counts, np.uint64).view(np.int64), "first": state["first"]}
        if out is not None:
            result["planes"] = out
        return result
    if kind == "stages":
        c, s, out = state["c"], state["s"], state["out"]
        base, m, v, t = state["parts"][0]
        s.reset_async(stream)
        P.stage_sim(c, v, t, m, out[0], out[1], stream)
        P.stage_mark(c, out[0], out[1], out[2], m, stream)
        P.stage_merge(c, s, out[0], out[2], m, base, stream)
        tot = P.stage_cover(c, s, out[2], m, base, stream)
        P.first_copy(s, state["first"][0], state["first"][1], False, stream)
        return {"count": np.array(_halves(tot), np.uint64).view(np.int64), "first": state["first"], "planes": out}
    if kind == "append":
        for _, s, *_ in state["jobs"]:
            s.reset_async(stream)
        for jobs in state["passes"]:
            state["batch"].rebind(jobs)
            state["batch"].run(stream)
    else:
        state["batch"].run(stream)
    totals = []
    for (c, s, *_), (fx, fy) in zip(state["jobs"], state["views"]):
        P.first_copy(s, fx, fy, False, stream)
        tot = P.Totals_t()
        P.check(P.lib().pdf_state_snapshot_on(s.h, None, None, ctypes.byref(tot), ctypes.c_void_p(stream)),
                "pdf_state_snapshot_on")
        totals.append(_halves(tot))
    return {"count": np.array(totals, np.uint64).view(np.int64), "first": state["first"]}


def work(case):
    """Bytes that a pass cannot do without: both code planes of the primary inputs read, two first-pair ids
    per net (or about two segments per net and extra level) written, and, when they are asked for, the two code
    planes and the mark plane of every net written."""
    if case["kind"] in ("batch", "append"):
        total = 0.0
        for gates, _, n in _members(case):
            total += max(16, gates // 13) * n / 4 + 8 * gates
        return {"bytes": total, "flops": 0.0}
    total = case["pio"] * case["pairs"] / 4 + 8 * case["gates"] * 2 ** (case.get("seg", 1) - 1)
    if case.get("planes") or case["kind"] == "stages":
        total += 3 * case["gates"] * case["pairs"] / 8
    return {"bytes": float(total), "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number or a plane of bits, which has to stay equal: none is a rounded value."""
    return None
