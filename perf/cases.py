"""Timed workloads of the engine through its public entry points.

``listed()`` holds the fixed workloads, ``draw(rng)`` gives another one of the
same ranges. ``prepare`` makes what a program has in hand before the call
(LPs, sessions, models, device buffers), ``run`` is one call or solve, ``work``
the bytes and operations it cannot do without, ``exact`` the same outputs in
64-bit arithmetic where they are plain linear algebra.

The single- and batched-LP workloads are planted LPs (columns of a given mean
degree, N(0,1) or log-uniform values, half equality rows, box bounds); the flow
workloads are min-cost flow on a fixed geometric graph with random supplies and
costs per instance, as in ``optimisation_solver_b200.generators``. The matrices
are built on the GPU here because the numpy generators take seconds at the
larger sizes.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from optimisation_solver_b200 import generators, native
from optimisation_solver_b200.learned import FlowWarmStart
from optimisation_solver_b200.lp import CompiledLp, PdlpOptions, SparseMatrix
from optimisation_solver_b200.mlp import Mlp, gemm_bf16
from optimisation_solver_b200.pdlp import PdlpSolver
from optimisation_solver_b200.session import Session

INF = float("inf")


def listed():
    return [
        # A toy model as a modelling layer sends it, one call per model: what a
        # call costs when the LP itself is nothing.
        dict(name="solve_tiny", kind="solve", rows=40, cols=70, degree=4, iterations=500,
             precision="fp64", tolerance=1e-6),
        # The drop-in call on the reference-sized LP (1000 x 2000, 4 per
        # column) at the reference's tolerance and arithmetic.
        dict(name="solve_1000x2000", kind="solve", rows=1000, cols=2000, degree=4,
             iterations=1500, precision="fp64", tolerance=1e-6),
        # One flow instance per call, the plain single-instance use of the
        # flow family (2000 nodes, 20,000 arcs).
        dict(name="solve_flow_2000", kind="solve_flow", nodes=2000, iterations=4600,
             precision="fp64", tolerance=1e-4),
        # A large LP whose costs change between solves: the session keeps the
        # matrix, each solve runs a fixed budget of 500 iterations (the
        # reference's 200k x 400k, 2M-nonzero benchmark).
        dict(name="resolve_200kx400k", kind="resolve", rows=200_000, cols=400_000, degree=5,
             family="normal", iterations=500, precision="fp64"),
        # A batch of independent LPs of very different sizes in one call.
        dict(name="batch_uneven_48", kind="batch", count=48, low=200, high=20_000,
             iterations=500, precision="mixed", tolerance=1e-4),
        # The throughput use: a stream of flow instances through 256 slots,
        # inputs and outputs in device memory, mixed precision.
        dict(name="flow_stream_256", kind="stream", nodes=2000, slots=256, count=512,
             iterations=4750, precision="mixed", tolerance=1e-4, device=True),
        # A smaller family served from host arrays in FP64.
        dict(name="flow_stream_fp64_48", kind="stream", nodes=500, slots=48, count=96,
             iterations=2500, precision="fp64", tolerance=1e-4, device=False),
        # One PDHG trial on device CSR arrays of the caller (the building
        # block for loops that own their memory).
        dict(name="trial_200kx400k", kind="trial", rows=200_000, cols=400_000, degree=5,
             family="normal"),
        # Training the learned warm start: four Adam steps on the flow
        # family's network (22,000 inputs, 22,016 outputs), weights read back.
        dict(name="train_flow_256", kind="train", inputs=22_000, hidden=512, outputs=22_016,
             batch=256, steps=4),
        # Predicting warm starts for one step's 256 instances: encode,
        # forward, decode.
        dict(name="predict_flow_256", kind="predict", nodes=2000, hidden=512, batch=256),
        # The BF16 GEMM alone at the size its throughput is quoted on, and a
        # ragged one with a K split.
        dict(name="gemm_8192", kind="gemm", m=8192, n=8192, k=8192, splits=1),
        dict(name="gemm_ragged", kind="gemm", m=1000, n=1544, k=2568, splits=4),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve_flow", "resolve", "resolve", "batch", "stream",
                       "trial", "trial", "train", "predict", "gemm", "gemm"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "solve":
        rows = _log_int(rng, 25, 4000)
        return dict(kind=kind, rows=rows, cols=rows + _log_int(rng, 10, 2 * rows),
                    degree=rng.randint(3, 8), iterations=1500, precision=precision,
                    tolerance=rng.choice([1e-4, 1e-6]))
    if kind == "solve_flow":
        return dict(kind=kind, nodes=_log_int(rng, 200, 2500), iterations=3500,
                    precision="fp64", tolerance=1e-4)
    if kind == "resolve":
        rows = _log_int(rng, 8000, 220_000)
        return dict(kind=kind, rows=rows, cols=rows + _log_int(rng, 1000, rows),
                    degree=rng.randint(3, 9), family=rng.choice(["normal", "zipf"]),
                    iterations=rng.randint(200, 500), precision=precision)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(5, 48), low=rng.randint(50, 500),
                    high=_log_int(rng, 2000, 20_000), iterations=500, precision=precision,
                    tolerance=1e-4)
    if kind == "stream":
        nodes = _log_int(rng, 150, 1500)
        slots = _log_int(rng, 4, 200)
        return dict(kind=kind, nodes=nodes, slots=slots, count=slots + rng.randint(1, slots),
                    iterations=3000, precision=precision, tolerance=1e-4,
                    device=rng.random() < 0.5)
    if kind == "trial":
        rows = _log_int(rng, 300, 220_000)
        return dict(kind=kind, rows=rows, cols=rows + _log_int(rng, 10, rows),
                    degree=rng.randint(2, 12), family=rng.choice(["normal", "zipf"]))
    if kind == "train":
        return dict(kind=kind, inputs=8 * _log_int(rng, 100, 2750),
                    hidden=64 * rng.randint(2, 8), outputs=64 * _log_int(rng, 10, 344),
                    batch=8 * _log_int(rng, 4, 32), steps=4)
    if kind == "predict":
        return dict(kind=kind, nodes=_log_int(rng, 150, 2000), hidden=64 * rng.randint(4, 8),
                    batch=8 * _log_int(rng, 4, 32))
    k = 8 * _log_int(rng, 16, 1000)
    return dict(kind=kind, m=_log_int(rng, 60, 8000), n=_log_int(rng, 60, 8000), k=k,
                splits=rng.choice([1, 1, 3, 8]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (seed % 1_000_000_007) + 12_345)
    return g


def _planted(gen, rows, cols, degree, family):
    """A feasible, bounded LP with a planted optimal pair; CSR of A on the host."""
    dev = "cuda"
    if family == "zipf":   # heavy-tailed column lengths, magnitudes over four decades
        u = torch.rand(cols, generator=gen, device=dev, dtype=torch.float64).clamp_min(1e-12)
        deg = (degree / 2.25 * u.pow(-1.0 / 1.8)).floor().clamp(1, min(1000, rows)).long()
    else:
        deg = torch.randint(max(1, degree - 2), degree + 3, (cols,), generator=gen, device=dev)
        deg = deg.clamp(max=rows)
    col = torch.repeat_interleave(torch.arange(cols, device=dev), deg)
    row = torch.randint(0, rows, (col.numel(),), generator=gen, device=dev)
    key = torch.unique(row * cols + col)
    row, col = key // cols, key % cols
    if family == "zipf":
        val = 10.0 ** (4.0 * torch.rand(key.numel(), generator=gen, device=dev, dtype=torch.float64) - 2.0)
        val *= torch.where(torch.rand(key.numel(), generator=gen, device=dev) < 0.5, -1.0, 1.0)
    else:
        val = torch.randn(key.numel(), generator=gen, device=dev, dtype=torch.float64)
    start = torch.zeros(rows + 1, dtype=torch.int64, device=dev)
    start[1:] = torch.cumsum(torch.bincount(row, minlength=rows), 0)
    ir, ic, v = row.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()

    def rand(n):
        return torch.rand(n, generator=gen, device=dev, dtype=torch.float64).cpu().numpy()

    def randn(n):
        return torch.randn(n, generator=gen, device=dev, dtype=torch.float64).cpu().numpy()

    upper = np.full(cols, 10.0) if family != "zipf" else 1.0 + 99.0 * rand(cols)
    kind, side = rand(cols), rand(cols)
    at_lower, at_upper = (kind >= 0.7) & (side < 0.5), (kind >= 0.7) & (side >= 0.5)
    x = np.where(at_lower, 0.0, np.where(at_upper, upper, rand(cols) * upper))
    b = np.bincount(ir, weights=v * x[ic], minlength=rows)
    equal = np.arange(rows) < rows // 2
    slack = ~equal & (rand(rows) < 0.5)
    y = randn(rows)
    y = np.where(equal, y, np.where(slack, 0.0, -np.abs(y)))
    row_upper = np.where(slack, b + rand(rows), b)
    row_lower = np.where(equal, b, -INF)
    z = np.abs(randn(cols))
    z = np.where(at_lower, z, np.where(at_upper, -z, 0.0))
    c = np.bincount(ic, weights=v * y[ir], minlength=cols) + z
    matrix = SparseMatrix(rows, cols, start.cpu().numpy(), ic.astype(np.int32), v)
    return CompiledLp(matrix, c, row_lower, row_upper, np.zeros(cols), upper, 0.0)


@functools.lru_cache(maxsize=4)
def _graph(nodes):
    """The flow family's graph (the same for every instance) and, per node, its
    incident arcs with their signs, padded to one length."""
    graph = generators.flow_graph(nodes, 5, seed=0)
    arcs = np.concatenate([np.arange(graph.arcs)] * 2)
    node = np.concatenate([graph.tail, graph.head])
    sign = np.concatenate([np.ones(graph.arcs), -np.ones(graph.arcs)])
    order = np.argsort(node, kind="stable")
    count = np.bincount(node, minlength=nodes)
    place = np.arange(order.size) - np.repeat(np.cumsum(count) - count, count)
    index = np.zeros((nodes, int(count.max())), dtype=np.int64)
    weight = np.zeros(index.shape)
    index[node[order], place] = arcs[order]
    weight[node[order], place] = sign[order]
    return graph, index, weight


def _flow_instances(gen, nodes, count):
    """Device FP64 (supply [count, nodes], cost [count, arcs]) of random instances."""
    graph, index, weight = _graph(nodes)
    dev = "cuda"
    index, weight = torch.as_tensor(index, device=dev), torch.as_tensor(weight, device=dev)
    capacity, length = torch.as_tensor(graph.capacity, device=dev), torch.as_tensor(graph.length, device=dev)
    flow = torch.rand((count, graph.arcs), generator=gen, device=dev, dtype=torch.float64) * capacity
    supply = torch.zeros((count, nodes), dtype=torch.float64, device=dev)
    for k in range(index.shape[1]):
        supply += flow[:, index[:, k]] * weight[:, k]
    noise = torch.randn((count, graph.arcs), generator=gen, device=dev, dtype=torch.float64)
    return graph, supply, length * torch.exp(0.2 * noise)


def _trial_inputs(case, seed):
    """The device arrays of one trial on an equilibrated LP, and the host LP."""
    gen = _generator(seed)
    lp = _planted(gen, case["rows"], case["cols"], case["degree"], case["family"])
    rows, cols = case["rows"], case["cols"]
    dev = "cuda"

    def put(a):
        return torch.as_tensor(np.ascontiguousarray(a), device=dev)

    ir = np.repeat(np.arange(rows), np.diff(lp.row_start))
    order = np.argsort(lp.col_index, kind="stable")
    at_start = np.zeros(cols + 1, dtype=np.int64)
    np.cumsum(np.bincount(lp.col_index, minlength=cols), out=at_start[1:])
    rs = np.bincount(ir, weights=np.abs(lp.values), minlength=rows)
    cs = np.bincount(lp.col_index, weights=np.abs(lp.values), minlength=cols)
    rs[rs == 0.0], cs[cs == 0.0] = 1.0, 1.0
    x = (torch.rand(cols, generator=gen, device=dev, dtype=torch.float64).cpu().numpy() * lp.var_upper)
    y = torch.randn(rows, generator=gen, device=dev, dtype=torch.float64).cpu().numpy()
    ax = np.bincount(ir, weights=lp.values * x[lp.col_index], minlength=rows)
    return dict(
        a_start=put(lp.row_start), a_index=put(lp.col_index), a_value=put(lp.values),
        at_start=put(at_start), at_index=put(ir[order].astype(np.int32)), at_value=put(lp.values[order]),
        c=put(lp.objective), xl=put(lp.var_lower), xu=put(lp.var_upper), tau=put(1.0 / cs), itau=put(cs),
        rl=put(lp.row_lower), ru=put(lp.row_upper), sigma=put(1.0 / rs), isigma=put(rs),
        x=put(x), y=put(y), ax=put(ax))


TRIAL_STEP, TRIAL_WEIGHT = 0.7, 1.3


def _network(case, seed):
    """He-initialised weights and one set of batches, on the device."""
    gen = _generator(seed)
    i, h, o, b = case["inputs"], case["hidden"], case["outputs"], case["batch"]

    def normal(*shape, std=1.0):
        return torch.randn(shape, generator=gen, device="cuda") * std

    params = dict(W1=normal(h, i, std=math.sqrt(2.0 / i)), b1=normal(h, std=0.01),
                  W2=normal(h, h, std=math.sqrt(2.0 / h)), b2=normal(h, std=0.01),
                  W3=normal(o, h, std=math.sqrt(2.0 / h)), b3=normal(o, std=0.01))
    batches = [(normal(b, i).to(torch.bfloat16), normal(b, o)) for _ in range(case.get("steps", 0))]
    return params, batches


def _predict_inputs(case, seed):
    """Instances, trained-looking weights and feature statistics of a predictor."""
    gen = _generator(seed)
    graph, supply, cost = _flow_instances(gen, case["nodes"], case["batch"])
    count = graph.nodes + graph.arcs
    sizes = dict(inputs=(count + 7) // 8 * 8, hidden=case["hidden"],
                 outputs=(count + 1 + 63) // 64 * 64, batch=case["batch"])
    params, _ = _network(sizes, seed + 1)
    feats = torch.cat([supply, cost], dim=1)
    mean, std = feats.mean(dim=0).float(), feats.std(dim=0).float().clamp_min(1e-6)
    ystd = torch.rand(graph.nodes, generator=gen, device="cuda") + 0.5
    ymean = torch.randn(graph.nodes, generator=gen, device="cuda")
    stats = dict(fmean=mean, finv=1.0 / std, ymean=ymean, ystd=ystd, yinv=1.0 / ystd,
                 wmean=0.3, wstd=0.4)
    return graph, supply, cost, params, stats


def _tolerance_options(case):
    # A budget that bounds the time of a hard draw; the listed solves end by
    # their tolerance well inside it.
    return PdlpOptions(iteration_limit=20_000).with_tolerance(case["tolerance"])


def prepare(case, seed):
    kind = case["kind"]
    state = dict(kind=kind, case=case)
    if kind == "solve":
        lp = _planted(_generator(seed), case["rows"], case["cols"], case["degree"], "normal")
        state.update(solver=PdlpSolver(case["precision"]), lp=lp, options=_tolerance_options(case))
    elif kind == "solve_flow":
        graph, supply, cost = _flow_instances(_generator(seed), case["nodes"], 1)
        lp = generators.flow_lp(graph, supply[0].cpu().numpy(), cost[0].cpu().numpy())
        state.update(solver=PdlpSolver(case["precision"]), lp=lp, options=_tolerance_options(case))
    elif kind == "resolve":
        gen = _generator(seed)
        lp = _planted(gen, case["rows"], case["cols"], case["degree"], case["family"])
        options = PdlpOptions(iteration_limit=case["iterations"], use_feasibility_polishing=False)
        options = options.with_tolerance(1e-12)
        cost = torch.as_tensor(lp.objective, device="cuda") * (
            1.0 + 0.1 * torch.rand(case["cols"], generator=gen, device="cuda", dtype=torch.float64))
        out = lambda n: torch.empty((1, n), dtype=torch.float64, device="cuda")  # noqa: E731
        state.update(session=Session(lp, 1, options, precision=case["precision"]),
                     cost=cost.reshape(1, -1), x=out(case["cols"]), y=out(case["rows"]))
    elif kind == "batch":
        gen = _generator(seed)
        # Rows evenly spread over the logarithm of the range, small and large in turn.
        sizes = np.exp(np.linspace(np.log(case["low"]), np.log(case["high"]), case["count"]))
        sizes = sizes[np.argsort(np.arange(case["count"]) * 7 % case["count"], kind="stable")]
        lps = [_planted(gen, int(m), 2 * int(m), 8, "normal") for m in sizes]
        state.update(solver=PdlpSolver(case["precision"]), lps=lps, options=_tolerance_options(case))
    elif kind == "stream":
        graph, supply, cost = _flow_instances(_generator(seed), case["nodes"], case["count"])
        family = generators.flow_lp(graph, supply[0].cpu().numpy(), cost[0].cpu().numpy())
        session = Session(family, case["slots"], _tolerance_options(case), precision=case["precision"])
        if case["device"]:
            x, y = torch.empty_like(cost), torch.empty_like(supply)
        else:
            supply, cost = supply.cpu().numpy(), cost.cpu().numpy()
            x, y = np.zeros_like(cost), np.zeros_like(supply)
        state.update(session=session, supply=supply, cost=cost, x=x, y=y)
    elif kind == "trial":
        a = _trial_inputs(case, seed)
        out = dict(x=torch.empty_like(a["x"]), y=torch.empty_like(a["y"]), ax=torch.empty_like(a["y"]),
                   red=torch.empty(3, dtype=torch.float64, device="cuda"))
        state.update(inputs=a, out=out)
    elif kind == "train":
        params, batches = _network(case, seed)
        mlp = Mlp(case["inputs"], case["hidden"], case["outputs"], case["batch"])
        mlp.set_params(params)
        weights = torch.full((case["outputs"],), 1.0 / case["outputs"], device="cuda")
        state.update(mlp=mlp, batches=batches, weights=weights,
                     params={k: torch.empty_like(v) for k, v in params.items()})
    elif kind == "predict":
        graph, supply, cost, params, stats = _predict_inputs(case, seed)
        model = FlowWarmStart(graph, hidden=case["hidden"], batch=case["batch"])
        model.mlp.set_params(params)
        model.stats = stats
        state.update(model=model, supply=supply, cost=cost)
    elif kind == "gemm":
        a, b = _gemm_inputs(case, seed)
        state.update(a=a, b=b, c=torch.empty((case["m"], case["n"]), device="cuda"))
    else:
        raise ValueError(kind)
    return state


def _gemm_inputs(case, seed):
    gen = _generator(seed)
    return (torch.randn((case["m"], case["k"]), generator=gen, device="cuda").to(torch.bfloat16),
            torch.randn((case["n"], case["k"]), generator=gen, device="cuda").to(torch.bfloat16))


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _solution(r):
    return dict(primal=r.primal, row_dual=r.row_dual, status=int(r.status), iterations=r.iterations,
                primal_objective=r.primal_objective, dual_objective=r.dual_objective)


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def run(state):
    kind = state["kind"]
    if kind in ("solve", "solve_flow"):
        return _solution(state["solver"].solve(state["lp"], state["options"]))
    if kind == "resolve":
        s = state["session"]
        s.load(objective=state["cost"], on_device=True)
        s.solve()
        r = s.read(primal=state["x"], dual=state["y"], on_device=True)
        return dict(primal=state["x"], dual=state["y"], iterations=r["iterations"],
                    primal_objective=r["primal_objective"])
    if kind == "batch":
        rs = state["solver"].solve_batch(state["lps"], state["options"])
        return dict(primal=np.concatenate([r.primal for r in rs]),
                    dual=np.concatenate([r.row_dual for r in rs]),
                    status=np.array([int(r.status) for r in rs]),
                    iterations=np.array([r.iterations for r in rs]),
                    objective=np.array([r.primal_objective for r in rs]))
    if kind == "stream":
        r = state["session"].stream(state["case"]["count"], objective=state["cost"],
                                    row_lower=state["supply"], row_upper=state["supply"],
                                    primal=state["x"], dual=state["y"],
                                    on_device=state["case"]["device"])
        return dict(primal=state["x"], dual=state["y"], iterations=r["iterations"],
                    status=np.array([int(s) for s in r["status"]]),
                    objective=r["primal_objective"])
    if kind == "trial":
        a, o = state["inputs"], state["out"]
        rc = native.lib().pdlpgpu_trial_noalloc(
            state["case"]["rows"], state["case"]["cols"], _ptr(a["a_start"]), _ptr(a["a_index"]),
            _ptr(a["a_value"]), _ptr(a["at_start"]), _ptr(a["at_index"]), _ptr(a["at_value"]),
            _ptr(a["c"]), _ptr(a["xl"]), _ptr(a["xu"]), _ptr(a["tau"]), _ptr(a["itau"]), _ptr(a["rl"]),
            _ptr(a["ru"]), _ptr(a["sigma"]), _ptr(a["isigma"]), _ptr(a["x"]), _ptr(a["y"]),
            _ptr(a["ax"]), TRIAL_STEP, TRIAL_WEIGHT, _ptr(o["x"]), _ptr(o["y"]), _ptr(o["ax"]),
            _ptr(o["red"]), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(native.last_error())
        return o
    if kind == "train":
        losses = [state["mlp"].train_step(x, t, state["weights"], 1e-3) for x, t in state["batches"]]
        state["mlp"].get_params(state["params"])
        return dict(losses=losses, params=state["params"])
    if kind == "predict":
        primal, dual, weight = state["model"].predict(state["supply"], state["cost"])
        return dict(primal=primal, dual=dual, weight=weight)
    gemm_bf16(state["a"], state["b"], state["c"], state["case"]["splits"])
    return state["c"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _iteration(rows, cols, nnz, batch, size):
    """Bytes of one PDHG iteration: both matrix passes (a matrix shared by the
    batch counts once), the iterates, bounds, costs and step vectors of each."""
    return 2 * nnz * (size + 4) + batch * size * (8 * cols + 9 * rows)


def work(case):
    kind = case["kind"]
    size = 4 if case.get("precision") == "mixed" else 8
    if kind in ("solve", "resolve"):
        nnz = case["degree"] * case["cols"]
        n = case["iterations"]
        return dict(bytes=n * _iteration(case["rows"], case["cols"], nnz, 1, size), flops=4.0 * n * nnz)
    if kind == "solve_flow":
        nodes, arcs, n = case["nodes"], 10 * case["nodes"], case["iterations"]
        return dict(bytes=n * _iteration(nodes, arcs, 2 * arcs, 1, size), flops=8.0 * n * arcs)
    if kind == "batch":
        mean = (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        rows, n = case["count"] * mean, case["iterations"]
        return dict(bytes=n * _iteration(rows, 2 * rows, 16 * rows, 1, size), flops=64.0 * n * rows)
    if kind == "stream":
        nodes, arcs = case["nodes"], 10 * case["nodes"]
        rounds = case["iterations"] * case["count"] / case["slots"]
        per = 2 * 2 * arcs * (size + 4) + case["slots"] * size * (5 * arcs + 8 * nodes)
        return dict(bytes=rounds * per, flops=8.0 * rounds * case["slots"] * arcs)
    if kind == "trial":
        rows, cols, nnz = case["rows"], case["cols"], case["degree"] * case["cols"]
        return dict(bytes=24.0 * nnz + 64.0 * cols + 88.0 * rows, flops=4.0 * nnz)
    if kind == "train":
        i, h, o, b = case["inputs"], case["hidden"], case["outputs"], case["batch"]
        p = h * (i + h + o)
        # FP32 weights and Adam moments read and written, the BF16 copies
        # written and read by both directions; at the end the weights copied out.
        step = 26 * p + 2 * (p + h * h + h * o) + b * (2 * i + 4 * o)
        return dict(bytes=case["steps"] * step + 8.0 * p,
                    flops=case["steps"] * 2.0 * b * (2 * h * i + 3 * h * h + 3 * h * o))
    if kind == "predict":
        n = 11 * case["nodes"]
        return dict(bytes=4.0 * n * case["hidden"] + 16.0 * case["batch"] * n,
                    flops=4.0 * case["batch"] * n * case["hidden"])
    m, n, k = case["m"], case["n"], case["k"]
    return dict(bytes=2.0 * k * (m + n) + 4.0 * m * n, flops=2.0 * m * n * k)


# ---------------------------------------------------------------------------
# The same in 64-bit arithmetic
# ---------------------------------------------------------------------------
def exact(case, seed):
    """None for the iterative solves (their outputs are where an iteration
    stopped) and for training (an Adam step divides by near-zero gradients)."""
    kind = case["kind"]
    if kind == "trial":
        a = _trial_inputs(case, seed)
        rows, cols = case["rows"], case["cols"]

        def product(start, index, value, v, n):
            line = torch.repeat_interleave(torch.arange(n, device="cuda"), start[1:] - start[:-1])
            p = (value * v[index.long()]).cpu().numpy()
            return torch.as_tensor(np.bincount(line.cpu().numpy(), weights=p, minlength=n), device="cuda")

        g = a["c"] + product(a["at_start"], a["at_index"], a["at_value"], a["y"], cols)
        x = torch.maximum(a["xl"], torch.minimum(a["x"] - TRIAL_STEP / TRIAL_WEIGHT * a["tau"] * g, a["xu"]))
        ax = product(a["a_start"], a["a_index"], a["a_value"], x, rows)
        step = TRIAL_STEP * TRIAL_WEIGHT * a["sigma"]
        v = a["y"] + step * (2.0 * ax - a["ax"])
        y = torch.clamp_min(v - step * a["ru"], 0.0) + torch.clamp_max(v - step * a["rl"], 0.0)
        dx, dy = x - a["x"], y - a["y"]
        red = torch.stack([(dx * dx * a["itau"]).sum(), (dy * dy * a["isigma"]).sum(),
                           (dy * (ax - a["ax"])).sum()])
        return dict(x=x, y=y, ax=ax, red=red)
    if kind == "predict":
        graph, supply, cost, p, stats = _predict_inputs(case, seed)
        feats = (torch.cat([supply, cost], dim=1) - stats["fmean"].double()) * stats["finv"].double()
        w = {k: v.double() for k, v in p.items()}
        h = torch.relu(feats @ w["W1"][:, :feats.shape[1]].T + w["b1"])
        h = torch.relu(h @ w["W2"].T + w["b2"])
        out = h @ w["W3"].T + w["b3"]
        n, m = graph.arcs, graph.nodes
        return dict(primal=out[:, :n].clamp(0.0, 1.0) * torch.as_tensor(graph.capacity, device="cuda"),
                    dual=out[:, n:n + m] * stats["ystd"].double() + stats["ymean"].double(),
                    weight=torch.exp(out[:, n + m] * stats["wstd"] + stats["wmean"]))
    if kind == "gemm":
        a, b = _gemm_inputs(case, seed)
        return a.double() @ b.double().T
    return None
