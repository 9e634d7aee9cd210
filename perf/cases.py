"""The work that a user of this framework has it do, for timing and for comparing results.

Six kinds of call, each through a public entry point of the Python binding:

  solve     Solver.run() and what a program then reads: the best individual, the fitness
            history, and the final population of a two-objective problem
  evaluate  Problem.evaluate_population on device buffers: the drop-in for a config's own
            evaluate_population_gpu
  step      one generation on device buffers: elite partition, generation step (crossover,
            mutants, decode, fitness), elite partition of the new population
  pareto    Pareto ranks (and crowding distances) of a pool of objective vectors
  batch     many island instances advanced together, from the batch's creation to its results
  serve     a stream of mixed solve requests through the server

Problem kinds: TSP (coordinates, matrix), bi-objective TSP, TSPJ, knapsack (threshold and
greedy decoders), job scheduling, continuous functions and the capacitated VRP.  Keys are
uniform on the 24-bit grid of [0, 1) that the engine and torch.rand both produce; everything
is float32, as the framework has no other key type.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-brkga_b200"))
import brkga_b200 as B  # noqa: E402

KINDS = ("tsp", "tsp_matrix", "bitsp", "tspj", "knap_threshold", "knap_greedy", "jobsched", "continuous", "movrp")
TWO_OBJECTIVES = ("bitsp", "movrp")
NO_ORDER = ("knap_threshold", "jobsched", "continuous")  # fitness straight from the keys, no argsort
BOUNDS = {0: (-5.12, 5.12), 1: (-5.12, 5.12), 2: (-5.0, 10.0)}  # sphere, Rastrigin, Rosenbrock


def listed():
    return [
        # the smallest whole solve: 52 cities, a population of 256, 500 generations; launches count
        dict(name="solve_tsp52", call="solve", kind="tsp", n=52, P=256, E=51, M=25, rho=0.7, gens=500),
        # the solver at scale: 1000 cities, a population of 2048, 1000 generations
        dict(name="solve_tsp1000", call="solve", kind="tsp", n=1000, P=2048, E=307, M=307, rho=0.7, gens=1000),
        # NSGA-II on a two-distance TSP, diversity pass every 25 generations
        dict(name="solve_bitsp500", call="solve", kind="bitsp", n=500, P=2048, E=0, M=204, rho=0.7, gens=250),
        # NSGA-II on a capacitated VRP, the population configure_for_size gives at 100 customers
        dict(name="solve_movrp100", call="solve", kind="movrp", n=100, P=1500, E=300, M=0, rho=0.10, gens=250),
        # TSPJ (tour and job assignment, two key segments) with its 2-opt local search
        dict(name="solve_tspj100", call="solve", kind="tspj", n=100, P=1000, E=200, M=100, rho=0.75, gens=500, ls=2),
        # a plugin's fitness call: the greedy knapsack at the largest size the server is asked for
        dict(name="eval_knapsack10000", call="evaluate", kind="knap_greedy", n=10000, P=1024, perm=False),
        # a plugin's fitness call: a continuous function in many variables
        dict(name="eval_rosenbrock1000", call="evaluate", kind="continuous", fn=2, n=1000, P=2048, perm=False),
        # a plugin's fitness call on the longest rows: they do not fit in shared memory
        dict(name="eval_tsp65536", call="evaluate", kind="tsp", n=65536, P=512, perm=False),
        # one generation of job scheduling on a program's own buffers
        dict(name="step_jobsched1000", call="step", kind="jobsched", n=1000, machines=32, P=2048, E=307, M=307, rho=0.7),
        # ranks and crowding of a pool of 2 x 2048 points
        dict(name="pareto4096", call="pareto", N=4096, dup=True),
        # 64 TSP instances of 100 .. 2000 cities, four islands each, migration on
        dict(name="batch64", call="batch", count=64, n_lo=100, n_hi=2000, gens=250, interval=50, migrants=2),
        # 24 mixed requests through the server: half TSP, 30 % greedy knapsack, 20 % bi-objective TSP
        dict(name="serve24", call="serve", count=24, gens=50, tick=25),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# chromosome lengths (cities, items, jobs, variables, customers) of each kind
LENGTHS = {"tsp": (20, 65536), "tsp_matrix": (20, 2000), "bitsp": (20, 5000), "tspj": (10, 500),
           "knap_threshold": (50, 10000), "knap_greedy": (50, 10000), "jobsched": (50, 3000),
           "continuous": (10, 1000), "movrp": (20, 500)}


def _ga(rng, P):
    return dict(E=max(1, int(P * rng.uniform(0.1, 0.25))), M=int(P * rng.uniform(0.0, 0.2)))


def _kind_options(rng, kind):
    if kind == "continuous":
        return dict(fn=rng.randrange(3))
    if kind == "jobsched":
        return dict(machines=_log(rng, 2, 100))
    return {}


def draw(rng):
    call = rng.choices(("solve", "evaluate", "step", "pareto", "batch", "serve"), (4, 4, 2, 1, 1, 1))[0]
    if call == "solve":
        kind = rng.choice(KINDS)
        lo, hi = LENGTHS[kind]
        n = _log(rng, lo, min(hi, 2000))
        P = _log(rng, 100, 2048)
        c = dict(call=call, kind=kind, n=n, P=P, rho=round(rng.uniform(0.6, 0.8), 2), gens=rng.randint(50, 250), **_ga(rng, P))
        if kind == "tspj" and rng.random() < 0.5:
            c["ls"] = 2
        return dict(c, **_kind_options(rng, kind))
    if call == "evaluate":
        kind = rng.choice(KINDS)
        lo, hi = LENGTHS[kind]
        n = _log(rng, lo, hi)
        P = min(_log(rng, 64, 8000), (1 << 25) // n)
        return dict(call=call, kind=kind, n=n, P=P, perm=kind not in NO_ORDER and rng.random() < 0.3,
                    **_kind_options(rng, kind))
    if call == "step":
        kind = rng.choice([k for k in KINDS if k not in TWO_OBJECTIVES])
        lo, hi = LENGTHS[kind]
        n = _log(rng, lo, min(hi, 20000))
        P = min(_log(rng, 100, 8000), (1 << 24) // n)
        return dict(call=call, kind=kind, n=n, P=P, rho=round(rng.uniform(0.6, 0.8), 2), **_ga(rng, P),
                    **_kind_options(rng, kind))
    if call == "pareto":
        return dict(call=call, N=_log(rng, 64, 8192), dup=rng.random() < 0.5)
    if call == "batch":
        return dict(call=call, count=rng.randint(4, 64), n_lo=100, n_hi=_log(rng, 300, 2000), gens=rng.randint(50, 250),
                    interval=rng.choice((10, 25, 50)), migrants=2)
    return dict(call=call, count=rng.randint(4, 24), gens=rng.randint(20, 50), tick=25)


# --------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------
def _instance(kind, n, rng, case):
    """the host arrays of one instance, as keyword arguments of Problem / Server.submit"""
    if kind == "tsp":
        return dict(kind=B.TSP_COORDS, n=n, coords=rng.random((n, 2), dtype=np.float32))
    if kind == "tsp_matrix":
        xy = rng.random((n, 2), dtype=np.float32)
        d = np.sqrt(((xy[:, None] - xy[None]) ** 2).sum(-1)).astype(np.float32)
        return dict(kind=B.TSP_MATRIX, n=n, matrix=d)
    if kind == "bitsp":
        return dict(kind=B.BITSP_COORDS, n=n, coords=rng.random((n + 1, 2), dtype=np.float32),
                    coords2=rng.random((n + 1, 2), dtype=np.float32))
    if kind == "tspj":
        # travel times: distances in [0, 100)^2; job durations 1 .. 100, the depot row zero
        xy = rng.random((n + 1, 2)) * 100.0
        travel = np.sqrt(((xy[:, None] - xy[None]) ** 2).sum(-1)).astype(np.float32)
        jobs = (1.0 + rng.random((n + 1, n + 1)) * 99.0).astype(np.float32)
        jobs[0] = 0.0
        return dict(kind=B.TSPJ, n=n, matrix=travel, matrix2=jobs)
    if kind in ("knap_threshold", "knap_greedy"):
        w = rng.integers(1, 101, n, dtype=np.int32)
        v = rng.integers(1, 101, n, dtype=np.int32)
        return dict(kind=B.KNAP_GREEDY if kind == "knap_greedy" else B.KNAP_THRESHOLD, n=n, weights=w, values=v,
                    capacity=float(np.float32(0.5 * float(w.sum()))))
    if kind == "jobsched":
        return dict(kind=B.JOBSCHED, n=n, machines=case["machines"],
                    job_times=(1.0 + rng.random(n) * 99.0).astype(np.float32))
    if kind == "continuous":
        lo, hi = BOUNDS[case["fn"]]
        return dict(kind=B.CONTINUOUS, n=n, function=case["fn"], lower=lo, upper=hi)
    # movrp: demands 1 .. 30, a fleet of n / 6 vehicles with ten per cent of slack
    dem = rng.integers(1, 31, n + 1).astype(np.int32)
    dem[0] = 0
    V = max(3, n // 6)
    return dict(kind=B.MOVRP, n=n, coords=(rng.random((n + 1, 2)) * 100.0).astype(np.float32), demands=dem,
                vehicle_capacity=max(30, int(math.ceil(1.1 * dem.sum() / V))), vehicles=V)


def _problem(case, seed):
    kw = _instance(case["kind"], case["n"], np.random.default_rng(seed), case)
    return kw, B.Problem(kw.pop("kind"), kw.pop("n"), **kw)


def _genes(case):
    return 2 * case["n"] if case["kind"] == "tspj" else case["n"]


def _keys(rows, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.randint(0, 1 << 24, (rows, n), device="cuda", generator=g, dtype=torch.int32)
    return k.to(torch.float32) * (1.0 / (1 << 24))


def _objectives(N, dup, seed):
    """a pool in mid-run: a convex trade-off curve with a spread of points behind it; with
    dup, a share of points listed twice, as survivor selection leaves them"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(N, device="cuda", generator=g)
    e = torch.rand(N, 2, device="cuda", generator=g)
    obj = torch.stack((20.0 + 15.0 * u, 20.0 + 15.0 * (1.0 - u.sqrt())), 1) + 4.0 * e
    if dup:
        q = N // 8
        obj[N - q:] = obj[:q]
    return obj.contiguous()


def _requests(case, seed):
    rng = np.random.default_rng(seed)
    reqs = []
    for i in range(case["count"]):
        u = (i + 0.5) / case["count"]
        if u < 0.5:
            n, kind, P, E, M = int(rng.integers(50, 5001)), "tsp", 512, 76, 76
        elif u < 0.8:
            n, kind, P, E, M = int(rng.integers(500, 10001)), "knap_greedy", 1024, 153, 153
        else:
            n, kind, P, E, M = 300, "bitsp", 512, 0, 51
        prm = B.params(P, E, M, 0.7, case["gens"], seed=seed * 1000 + i)
        reqs.append((dict(_instance(kind, n, rng, case)), prm))
    return reqs


def _batch_sizes(case, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(case["n_lo"], case["n_hi"] + 1, case["count"]), rng.choice([256, 512, 1024], case["count"])


def prepare(case, seed):
    call = case["call"]
    s = dict(case=case)
    if call == "solve":
        _, s["problem"] = _problem(case, seed)
        extra = dict(local_search_interval=case["ls"]) if case.get("ls") else {}
        s["solver"] = B.Solver(s["problem"], B.params(case["P"], case["E"], case["M"], case["rho"], case["gens"],
                                                      seed=seed + 1, **extra))
    elif call == "evaluate":
        _, s["problem"] = _problem(case, seed)
        s["pop"] = _keys(case["P"], _genes(case), seed)
        s["fit"] = torch.empty((case["P"], 2) if case["kind"] in TWO_OBJECTIVES else (case["P"],), device="cuda")
        s["perm"] = torch.empty(case["P"], _genes(case), dtype=torch.int32, device="cuda") if case["perm"] else None
    elif call == "step":
        _, s["problem"] = _problem(case, seed)
        P, n = case["P"], _genes(case)
        ld = (n + 3) // 4 * 4
        s["ld"], s["seed"] = ld, seed
        s["pop"] = torch.zeros(P, ld, device="cuda")
        s["pop"][:, :n] = _keys(P, n, seed)
        s["fit"] = torch.empty(P, device="cuda")
        s["problem"].evaluate_population(s["pop"], s["fit"], P, n, ld)
        s["next"], s["next_fit"] = torch.zeros_like(s["pop"]), torch.empty_like(s["fit"])
        s["order"] = torch.empty(P, dtype=torch.int32, device="cuda")
        s["next_order"] = torch.empty_like(s["order"])
    elif call == "pareto":
        s["obj"] = _objectives(case["N"], case["dup"], seed)
        s["rank"] = torch.empty(case["N"], dtype=torch.int32, device="cuda")
        s["cd"] = torch.empty(case["N"], device="cuda")
    elif call == "batch":
        ns, Ps = _batch_sizes(case, seed)
        s["problems"], s["params"] = [], []
        for i, (n, P) in enumerate(zip(ns, Ps)):
            s["problems"].append(B.tsp(np.random.default_rng([seed, i]).random((int(n), 2), dtype=np.float32)))
            s["params"].append(B.params(int(P), int(0.15 * P), int(0.15 * P), 0.7, case["gens"], seed=seed + i,
                                        num_islands=4, migration_interval=case["interval"],
                                        num_migrants=case["migrants"]))
    else:
        s["requests"] = _requests(case, seed)
        s["server"] = B.Server(generations_per_tick=case["tick"])
    return s


# --------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    call = case["call"]
    if call == "solve":
        solver = s["solver"]
        solver.run()
        keys, perm, fit = solver.get_best_individual()
        out = dict(keys=keys, fit=np.asarray(fit), history=solver.get_fitness_history())
        if case["kind"] not in NO_ORDER:
            out["perm"] = perm
        if case["kind"] in TWO_OBJECTIVES:
            out["population"], out["objectives"] = solver.get_population()
        return out
    if call == "evaluate":
        s["problem"].evaluate_population(s["pop"], s["fit"], case["P"], d_perm=s["perm"])
        return dict(fit=s["fit"], perm=s["perm"]) if case["perm"] else dict(fit=s["fit"])
    if call == "step":
        P, mx = case["P"], case["kind"].startswith("knap")
        B.sort_fitness(s["fit"], P, 1, mx, s["order"])
        B.generation_step(s["problem"], s["pop"], s["fit"], s["order"], s["next"], s["next_fit"], P, case["E"], case["M"],
                          case["rho"], s["ld"], s["seed"], 1)
        B.sort_fitness(s["next_fit"], P, 1, mx, s["next_order"])
        return dict(pop=s["next"], fit=s["next_fit"], order=s["next_order"])
    if call == "pareto":
        B.pareto_rank(s["obj"], case["N"], 2, s["rank"])
        if case["N"] > 4096:  # the crowding operator's limit
            return dict(rank=s["rank"])
        B.crowding(s["obj"], s["rank"], case["N"], 2, s["cd"])
        return dict(rank=s["rank"], cd=s["cd"])
    if call == "batch":
        batch = B.Batch(s["problems"], s["params"])  # a batch runs its members' generations once
        batch.evolve(case["gens"])
        best = batch.best()
        batch.close()
        return dict(best=best)
    server = s["server"]
    ids = [server.submit(prm=prm, **kw) for kw, prm in s["requests"]]
    done = {}
    while len(done) < len(ids):
        server.step()
        for i in ids:
            if i not in done:
                r = server.poll(i)
                if r is not None:
                    done[i] = r
    return dict(best=np.stack([done[i][1] for i in ids]), gens=np.array([done[i][2] for i in ids]),
                status=np.array([done[i][0] for i in ids]))


# --------------------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------------------
def _instance_bytes(kind, n, case):
    return {"tsp": 8 * n, "tsp_matrix": 4 * n * n, "bitsp": 16 * (n + 1), "tspj": 8 * (n + 1) ** 2, "knap_threshold": 8 * n,
            "knap_greedy": 8 * n, "jobsched": 4 * n, "continuous": 16, "movrp": 12 * (n + 1)}[kind]


# operations per gene: the terms of the sums, and log2(n) compares per key of an argsort
def _gene_ops(kind, n):
    terms = {"tsp": 6, "tsp_matrix": 1, "bitsp": 12, "tspj": 2, "knap_threshold": 3, "knap_greedy": 3, "jobsched": 2,
             "continuous": 6, "movrp": 14}[kind]
    return terms + (0 if kind in NO_ORDER else math.log2(max(2, n)))


def _generation_bytes(P, E, M, n, two):
    """elite rows read and written, an inherited gene read and one written for every child
    gene, mutant rows written (two objectives: P children, P survivors read and written)"""
    if two:
        return P * n * 4 * 4
    return 4 * n * (2 * E + 2 * (P - E - M) + M) + 8 * P


def work(case):
    call = case["call"]
    if call == "pareto":
        N = case["N"]
        return {"bytes": 8 * N + 4 * N + (4 * N if N <= 4096 else 0), "flops": 2 * N * math.log2(max(2, N))}
    if call == "batch":
        ns, Ps = _batch_sizes(case, 1)
        b = sum(_generation_bytes(int(P), int(0.15 * P), int(0.15 * P), int(n), False) for n, P in zip(ns, Ps))
        f = sum(int(P) * 0.85 * int(n) * _gene_ops("tsp", int(n)) for n, P in zip(ns, Ps))
        return {"bytes": case["gens"] * b, "flops": case["gens"] * f}
    if call == "serve":
        b = f = 0.0
        for kw, prm in _requests(case, 1):
            kind = {B.TSP_COORDS: "tsp", B.KNAP_GREEDY: "knap_greedy", B.BITSP_COORDS: "bitsp"}[kw["kind"]]
            P, n = prm.population_size, kw["n"]
            b += case["gens"] * _generation_bytes(P, prm.elite_size, prm.mutant_size, n, kind == "bitsp")
            f += case["gens"] * (P - prm.elite_size) * n * _gene_ops(kind, n)
        return {"bytes": b, "flops": f}
    kind, P, n = case["kind"], case["P"], _genes(case)
    two = kind in TWO_OBJECTIVES
    if call == "evaluate":
        return {"bytes": P * n * 4 * (2 if case["perm"] else 1) + P * 4 * (2 if two else 1) + _instance_bytes(kind, case["n"], case),
                "flops": P * n * _gene_ops(kind, n)}
    gens = case["gens"] if call == "solve" else 1
    E = 0 if two else case["E"]
    return {"bytes": gens * _generation_bytes(P, E, case["M"], n, two) + _instance_bytes(kind, case["n"], case),
            "flops": gens * (P - E) * n * _gene_ops(kind, n)}


# --------------------------------------------------------------------------------------
# the same results in 64 bits (evaluate and pareto; a run's and a step's populations follow
# the framework's own random stream and have no other source)
# --------------------------------------------------------------------------------------
def _exact_ranks(obj):
    """peeling in which the first front counts twice (the reference lists it twice)"""
    le = (obj[:, None, :] <= obj[None, :, :]).all(-1)
    lt = (obj[:, None, :] < obj[None, :, :]).any(-1)
    dom = le & lt  # dom[i, j]: i dominates j
    left = dom.sum(0)
    rank = torch.full((obj.shape[0],), -1, dtype=torch.int64, device=obj.device)
    r, front = 0, left == 0
    while bool(front.any()):
        rank[front] = r
        left = left - dom[front].sum(0) * (2 if r == 0 else 1)
        front = (left <= 0) & (rank < 0)
        r += 1
    return rank.cpu().numpy()


def _exact_crowding(obj, rank):
    cd = np.zeros(len(rank))
    for r in range(rank.max() + 1):
        idx = np.flatnonzero(rank == r)
        lst = np.repeat(idx, 2) if r == 0 else idx  # first-front points are listed twice
        if len(lst) <= 2:
            cd[lst] = np.inf
            continue
        for o in range(2):
            lst = lst[np.lexsort((lst, obj[lst, o]))]
            v = obj[lst, o]
            cd[lst[[0, -1]]] = np.inf
            if v[-1] > v[0]:
                np.add.at(cd, lst[1:-1], (v[2:] - v[:-2]) / (v[-1] - v[0]))
    return cd


def _exact_fitness(case, seed):
    kind, n, P = case["kind"], case["n"], case["P"]
    kw = _instance(kind, n, np.random.default_rng(seed), case)
    keys = _keys(P, _genes(case), seed)

    def t64(a):
        return torch.from_numpy(np.asarray(a)).to("cuda").double()

    if kind == "continuous":
        x = keys.double() * (float(np.float32(kw["upper"])) - float(np.float32(kw["lower"]))) + float(np.float32(kw["lower"]))
        if case["fn"] == 0:
            return (x * x).sum(1)
        if case["fn"] == 1:
            return 10.0 * n + (x * x - 10.0 * torch.cos(2.0 * math.pi * x)).sum(1)
        return (100.0 * (x[:, 1:] - x[:, :-1] ** 2) ** 2 + (1.0 - x[:, :-1]) ** 2).sum(1)
    if kind == "jobsched":
        M = case["machines"]
        where = (keys * float(M)).to(torch.int64).clamp_(0, M - 1)  # the machine is chosen in float32
        loads = torch.zeros(P, M, dtype=torch.float64, device="cuda")
        loads.scatter_add_(1, where, t64(kw["job_times"]).expand(P, n).contiguous())
        return loads.amax(1)
    if kind == "knap_threshold":
        take = (keys > 0.5).double()
        w, v, cap = take @ t64(kw["weights"]), take @ t64(kw["values"]), float(np.float32(kw["capacity"]))
        return torch.where(w > cap, v - (w - cap) * 1000.0, v)
    if kind == "tspj":
        city, job = (torch.sort(k, dim=1, stable=True).indices + 1 for k in (keys[:, :n], keys[:, n:]))
        travel, jobs = t64(kw["matrix"]), t64(kw["matrix2"])
        prev = torch.cat((torch.zeros_like(city[:, :1]), city[:, :-1]), 1)
        at = torch.cumsum(travel[prev, city], 1)
        return torch.maximum(at[:, -1] + travel[city[:, -1], 0], (at + jobs[city, job]).amax(1))
    perm = torch.sort(keys, dim=1, stable=True).indices
    if kind == "tsp":
        p = t64(kw["coords"])[perm]
        return (p - p.roll(-1, 1)).square().sum(-1).sqrt().sum(1)
    if kind == "tsp_matrix":
        return t64(kw["matrix"])[perm, perm.roll(-1, 1)].sum(1)
    if kind == "bitsp":
        depot = torch.zeros_like(perm[:, :1])
        tour = torch.cat((depot, perm + 1, depot), 1)
        ps = [t64(kw[c])[tour] for c in ("coords", "coords2")]
        return torch.stack([(p[:, 1:] - p[:, :-1]).square().sum(-1).sqrt().sum(1) for p in ps], 1)
    if kind == "knap_greedy":
        # items in key order, each taken when it still fits
        w, v = (torch.from_numpy(kw[c]).to("cuda").to(torch.int64)[perm].t().contiguous().cpu().numpy() for c in ("weights", "values"))
        room, value = np.full(P, int(math.floor(kw["capacity"]))), np.zeros(P, np.int64)
        for k in range(n):
            take = w[k] <= room
            room -= w[k] * take
            value += v[k] * take
        return torch.from_numpy(value.astype(np.float64))
    return None  # movrp: its decode order depends on float32 sums of the keys


def exact(case, seed):
    if case["call"] == "evaluate":
        fit = _exact_fitness(case, seed)
        if fit is None:
            return None
        return dict(fit=fit, perm=None) if case["perm"] else dict(fit=fit)
    if case["call"] == "pareto" and case["N"] <= 4096:
        obj = _objectives(case["N"], case["dup"], seed)
        return dict(rank=None, cd=_exact_crowding(obj.double().cpu().numpy(), _exact_ranks(obj)))
    return None
