"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is one of five kinds:
  infer    one request to a model executor: the input is copied from pinned host memory, the model
           runs, the result is copied back and waited for (the request pipeline of the clients).
           Latency-critical tenants use the base executor with a captured graph, best-effort tenants
           the preemptible executor; lists of more than 64 kernels are launched kernel by kernel, as
           the scheduler does with best-effort tenants, shorter ones as a graph.
  gemm     the preemptible bf16 GEMM (tensor-bound best-effort kernel)
  axpy     the preemptible fp32 axpy (memory-bound best-effort kernel)
  weather  miniWeather: initial conditions in, ten time steps, state out
  graph    one run of a graph-analytics workload on a graph that was loaded before

Inputs are made from the seed; weights are those of a fixed seed, loaded once and kept, as a serving
process keeps them.
"""
import ctypes
import json
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from gpreempt_b200 import api, graph_files
from gpreempt_b200 import binding

WEIGHT_SEED = 1
WEATHER_STEPS = 10


def listed():
    return [
        # A small vector of odd length through the preemptible axpy: launch latency.
        {"name": "axpy-1000003", "kind": "axpy", "n": 1000003},
        # The tensor-bound best-effort kernel of the preemption benchmark.
        {"name": "gemm-8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192},
        # The latency-critical tenant of the headline benchmark.
        _infer("resnet50", 1, "float32", hp=True),
        # The smallest latency-critical convolution model of the multi-tenant mix.
        _infer("mobilenet_v2", 1, "bfloat16", hp=True),
        # The latency-critical sequence model.
        _infer("bert_base", 1, "float16", hp=True, seq=128),
        # The sequence model of the task configurations at its six tokens.
        _infer("distilbert", 1, "float32", hp=True, seq=6),
        # Best-effort tenants: the headline benchmark's, and those of the other configurations.
        _infer("resnet50", 32, "float32"),
        _infer("vgg16", 16, "float16"),
        _infer("densenet201", 64, "bfloat16"),
        _infer("bert_base", 32, "bfloat16", seq=512),
        # The scientific best-effort tenant on its own grid.
        {"name": "miniweather-3200x1600", "kind": "weather", "nx": 3200, "nz": 1600},
        # The longest of the graph-analytics tenants on a graph of the size they are configured for.
        {"name": "pagerank-52804", "kind": "graph", "algo": "pagerank", "vertices": 52804, "degree": 201, "band": 1500},
    ]


def _infer(model, batch, dtype, hp=False, seq=0):
    name = "%s-b%d%s-%s" % (model, batch, "-s%d" % seq if seq else "", dtype)
    return {"name": name, "kind": "infer", "model": model, "batch": batch, "dtype": dtype, "seq": seq, "hp": hp}


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


# Largest batch drawn: it keeps a request below the largest listed one in time.
DRAWN_BATCH = {"resnet50": 64, "resnet152": 24, "vgg16": 24, "vgg19": 24, "mobilenet_v2": 64, "densenet201": 48,
               "inception_v3": 24, "bert_base": 32, "distilbert": 48}


def draw(rng):
    kind = rng.choice(["infer"] * 6 + ["gemm", "axpy", "weather", "graph"])
    if kind == "axpy":
        return {"kind": "axpy", "n": _log_int(rng, 1, 1 << 28)}
    if kind == "gemm":
        # whole tiles of 128 x 256 x 64, as the entry point requires
        return {"kind": "gemm", "m": 128 * _log_int(rng, 1, 64), "n": 256 * _log_int(rng, 1, 32), "k": 64 * _log_int(rng, 1, 128)}
    if kind == "weather":
        return {"kind": "weather", "nx": _log_int(rng, 100, 3200), "nz": _log_int(rng, 50, 1600)}
    if kind == "graph":
        return {"kind": "graph", "algo": rng.choice(["bfs", "sssp", "cc", "pagerank"]), "vertices": _log_int(rng, 3000, 52804),
                "degree": rng.randint(20, 201), "band": rng.randint(300, 1500)}
    model = rng.choice(sorted(DRAWN_BATCH))
    dtype = rng.choice(["float32", "bfloat16", "float16"])
    # latency-critical requests have batch 1 or a few, best-effort ones any
    hp = rng.random() < 0.4
    batch = _log_int(rng, 1, 4 if hp else DRAWN_BATCH[model])
    seq = 0
    if model == "bert_base":
        seq = 8 * _log_int(rng, 1, 64)
    elif model == "distilbert":
        seq = _log_int(rng, 4, 512) if dtype == "float32" else 8 * _log_int(rng, 1, 64)
    case = _infer(model, batch, dtype, hp, seq)
    del case["name"]
    return case


# ---- preparation ---------------------------------------------------------------------------------

_ready = {}


def _stream(priority):
    """One stream per priority class, as a client has (0 = latency-critical, 1 = best-effort)."""
    if "init" not in _ready:
        api.init_cuda(0)
        _ready["init"] = True
    if priority not in _ready:
        _ready[priority] = api.Stream(priority)
    return _ready[priority]


def _word():
    """The preempt word the best-effort work of this GPU shares; nobody raises it here."""
    if "word" not in _ready:
        _ready["word"] = api.PreemptWord(binding.WORD_DEVICE)
    return _ready["word"]


class _Tenant:
    """An executor with its model and weights; freed with its last user."""

    def __init__(self, case):
        self.stream = _stream(0 if case.get("hp") else 1)
        self.blp = not case.get("hp")
        self.ex = api.BLPExecutor() if self.blp else api.BaseExecutor()

    def start(self, graph):
        if self.blp:
            self.ex.set_word(_word())
        if graph:
            self.ex.capture_graph(self.stream)

    def execute(self):
        self.ex.execute(self.stream)

    def finish(self):
        """Waits; a preemptible executor's client reads the stop point, a base executor's just waits."""
        if self.blp:
            if self.ex.getStopPoint(self.stream) != -1:
                raise RuntimeError("stopped, although nobody raised the word")
        else:
            self.stream.sync()

    def __del__(self):
        try:
            self.ex.clear()
        except Exception:
            pass


def _kept_tenant(case, build):
    """The tenant of a case: its weights stay loaded while requests with other inputs come."""
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    kept = _ready.get("tenant")
    if kept is None or kept[0] != key:
        _ready["tenant"] = kept = None  # frees the previous case's model first, if no state holds it
        _ready["tenant"] = kept = (key, build(case))
    return kept[1]


def _build_infer(case):
    t = _Tenant(case)
    t.ex.init(case["model"], batch=case["batch"], seed=WEIGHT_SEED, seq_len=case["seq"], dtype=case["dtype"])
    t.start(graph=not t.blp or t.ex.get_kernel_num() <= 64)
    return t


def _build_weather(case):
    t = _Tenant(case)
    t.ex.init("miniweather_%dx%d" % (case["nx"], case["nz"]))
    t.start(graph=True)
    t.initial = t.ex.model.get("state")
    return t


def _pinned(shape, dtype):
    return torch.empty(tuple(int(v) for v in shape), dtype=dtype, pin_memory=True)


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


class _Ref:
    """A tensor's memory where the entry points take a device buffer."""

    def __init__(self, t):
        self.tensor = t
        self.ptr = ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind = case["kind"]
    s = _stream(0 if case.get("hp") else 1)
    g = _rng(seed)
    if kind == "axpy":
        x = torch.rand(case["n"], generator=g, device="cuda") * 2 - 1
        y = torch.rand(case["n"], generator=g, device="cuda") * 2 - 1
        return {"case": case, "x": _Ref(x), "y": _Ref(y), "blp": api.BlpContext(_word(), kernel_id=0, trace=False), "stream": s}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        a = (torch.rand(m, k, generator=g, device="cuda") * 2 - 1).bfloat16()
        b = (torch.rand(n, k, generator=g, device="cuda") * 2 - 1).bfloat16()
        return {"case": case, "a": _Ref(a), "b": _Ref(b), "c": _Ref(torch.empty(m, n, dtype=torch.bfloat16, device="cuda")),
                "ctx": api.GemmContext(), "blp": api.BlpContext(_word(), kernel_id=0, trace=False), "stream": s}
    if kind == "infer":
        t = _kept_tenant(case, _build_infer)
        shape = t.ex.model.shape("data")
        if "bert" in case["model"]:
            data = _pinned(shape, torch.int64)
            data.copy_(torch.randint(0, 30522, tuple(shape), generator=g, device="cuda"))
        else:
            data = _pinned(shape, torch.float32)
            data.copy_(torch.randn(tuple(shape), generator=g, device="cuda"))
        return {"case": case, "tenant": t, "in": data, "out": _pinned(t.ex.model.shape("heads"), torch.float32)}
    if kind == "weather":
        t = _kept_tenant(case, _build_weather)
        nx, nz = case["nx"], case["nz"]
        state = torch.from_numpy(t.initial).reshape(4, nz + 4, nx + 4).cuda()
        # a warm bubble somewhere in the domain, on the interior cells of the initial state
        cx, cz, size = (torch.rand(3, generator=g, device="cuda") * torch.tensor([0.6, 0.4, 0.1], device="cuda")
                        + torch.tensor([0.2, 0.2, 0.05], device="cuda")).tolist()
        xs = (torch.arange(nx, device="cuda") + 0.5) / nx - cx
        zs = (torch.arange(nz, device="cuda") + 0.5) / nz - cz
        bump = torch.exp(-(zs[:, None] ** 2 + xs[None, :] ** 2) / (2 * size * size))
        state[3, 2:2 + nz, 2:2 + nx] += 3.0 * bump
        pinned = _pinned(state.shape, torch.float32)
        pinned.copy_(state)
        return {"case": case, "tenant": t, "in": pinned, "out": _pinned(state.shape, torch.float32)}
    # graph: the files are written and loaded here; a run starts from the algorithm's initial state
    folder = tempfile.mkdtemp(prefix="graph_")
    try:
        prefix = os.path.join(folder, "g.bel")
        _write_graph(prefix, case, g)
        t = _Tenant(case)
        t.ex.set_graph_path(prefix)
        t.ex.init(case["algo"])
        t.start(graph=True)
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    result = {"bfs": "label", "sssp": "cost", "cc": "comp", "pagerank": "value"}[case["algo"]]
    out = _pinned((case["vertices"],), torch.float32 if result == "value" else torch.int32)
    return {"case": case, "tenant": t, "result": result, "out": out}


def _write_graph(prefix, case, g):
    """A symmetric banded graph, as a bandwidth-reduced mesh is: every vertex is tied to `degree`
    others within `band` of its own index, and to its successor."""
    v, half = case["vertices"], max(1, case["degree"] // 2)
    src = torch.arange(v, device="cuda").repeat_interleave(half)
    dst = src + torch.randint(1, case["band"] + 1, (v * half,), generator=g, device="cuda") * (
        torch.randint(0, 2, (v * half,), generator=g, device="cuda") * 2 - 1)
    inside = (dst >= 0) & (dst < v)
    chain = torch.arange(v - 1, device="cuda")
    src, dst = torch.cat([src[inside], chain]), torch.cat([dst[inside], chain + 1])
    key = torch.unique(torch.cat([src * v + dst, dst * v + src]))
    offsets = np.zeros(v + 1, np.uint64)
    offsets[1:] = torch.cumsum(torch.bincount(key // v, minlength=v), 0).cpu().numpy()
    neighbours = (key % v).cpu().numpy()
    weights = torch.randint(1, 65, (len(neighbours),), generator=g, device="cuda").cpu().numpy() if case["algo"] == "sssp" else None
    graph_files.write_bel(prefix, offsets, neighbours, weights)


# ---- one pass ------------------------------------------------------------------------------------

def _set(t, name, host):
    binding.check(binding.load().gpx_model_set(t.ex.model.handle, name, host.data_ptr(), host.nbytes, t.stream.handle))


def _get(t, name, host):
    binding.check(binding.load().gpx_model_get(t.ex.model.handle, name, host.data_ptr(), host.nbytes, t.stream.handle))


def run(state):
    case = state["case"]
    kind, s = case["kind"], state.get("stream")
    if kind == "axpy":
        # y is updated in place, pass after pass; the context is re-armed only after the pass before
        # it has ended, so a pass waits for itself
        state["blp"].reset()
        api.axpy(1.0009765625, state["x"], state["y"], case["n"], state["blp"], s)
        s.sync()
        return state["y"].tensor
    if kind == "gemm":
        state["ctx"].reset()
        state["blp"].reset()
        api.gemm_bf16(state["a"], state["b"], state["c"], case["m"], case["n"], case["k"], state["ctx"], state["blp"], s)
        s.sync()
        return state["c"].tensor
    t = state["tenant"]
    if kind == "infer":
        _set(t, b"data", state["in"])
        t.execute()
        _get(t, b"heads", state["out"])
        t.finish()
        return state["out"]
    if kind == "weather":
        _set(t, b"state", state["in"])
        for _ in range(WEATHER_STEPS):
            t.execute()
        _get(t, b"state", state["out"])
        t.finish()
        return state["out"]
    t.execute()
    _get(t, state["result"].encode(), state["out"])
    t.finish()
    return state["out"]


# ---- what a pass cannot do without ---------------------------------------------------------------

# millions of multiplications per image, millions of parameters
CONV_MODELS = {"resnet50": (4089.2, 25.5), "resnet152": (11513.6, 60.1), "vgg16": (15470.3, 138.4), "vgg19": (19632.1, 143.7),
               "mobilenet_v2": (300.8, 3.5), "densenet201": (4291.4, 19.8), "inception_v3": (5713.2, 23.8)}


def work(case):
    kind = case["kind"]
    if kind == "axpy":
        # x and y read, y written
        return {"bytes": 12 * case["n"], "flops": 2 * case["n"]}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if kind == "weather":
        # state in, state out; about 100 operations for each cell of each of the 12 passes of a step
        return {"bytes": 2 * 16 * (case["nx"] + 4) * (case["nz"] + 4), "flops": 100 * 12 * WEATHER_STEPS * case["nx"] * case["nz"]}
    if kind == "graph":
        edges = case["vertices"] * case["degree"]
        return {"bytes": (8 if case["algo"] == "sssp" else 4) * edges + 12 * case["vertices"], "flops": 2 * edges}
    b, elem = case["batch"], 4 if case["dtype"] == "float32" else 2
    if case["model"] in CONV_MODELS:
        mult, params = CONV_MODELS[case["model"]]
        pixels = 3 * (299 if case["model"] == "inception_v3" else 224) ** 2
        return {"bytes": params * 1e6 * elem + 4 * b * (pixels + 1000), "flops": 2e6 * mult * b}
    layers, rows = 12 if case["model"] == "bert_base" else 6, b * case["seq"]
    per_layer = 12 * 768 * 768
    return {"bytes": layers * per_layer * elem + rows * (8 + 4 * 768 + 4 * 768),
            "flops": 2 * layers * rows * (per_layer + 2 * case["seq"] * 768)}


def tolerance(case):
    kind = case["kind"]
    if kind == "axpy" or (kind == "graph" and case["algo"] != "pagerank"):
        return "exact"
    if kind == "gemm":
        return {"rel": 4e-3}  # one rounding to bf16
    if kind == "weather":
        return {"rel": 1e-5}
    if kind == "graph":
        return {"rel": 1e-4}  # a residual that meets the threshold in one order of summation and not in another
    # float32 models keep 16 bits of mantissa between layers; the 16-bit formats round every layer
    return {"rel": {"float32": 1e-4, "float16": 5e-3, "bfloat16": 1e-2}[case["dtype"]]}
