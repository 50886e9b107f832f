"""Sizes at which the layer kernels change form: edges of tiles, remainders, both sides of each limit."""
import numpy as np
import pytest

from gpreempt_b200 import graph_files

pytestmark = pytest.mark.gpu

TOL = {"float32": 1e-4, "float16": 5e-3, "bfloat16": 2e-2}  # of the largest value of a tensor


def _rel(a, b):
    return float(np.max(np.abs(a.astype(np.float64) - b.astype(np.float64))) / max(float(np.max(np.abs(b))), 1e-30))


def _images(gpx, batch, seed=0):
    return gpx.synth_normal(batch * 3 * 224 * 224, seed, 0).reshape(batch, 3, 224, 224)


def _bert(gpx, oracle, batch, seq, dtype):
    """bert_tiny on seeded ids: the executor after one forward, and the oracle's tensors."""
    ex = gpx.BaseExecutor()
    ex.init("bert_tiny", batch=batch, seed=7, seq_len=seq, dtype=dtype)
    ids = np.random.default_rng(seq).integers(0, 1000, (batch, seq)).astype(np.int64)
    ex.set_input("data", ids)
    ex.execute()
    assert ex.error() == (0, 0)
    params = {k: v.reshape(v.shape[0], -1) if v.ndim == 4 else v for k, v in ex.model.params().items()}
    taps = {}
    heads = oracle.bert_forward(params, ids, layers=2, heads=2, taps=taps)
    return ex, taps, heads


# One block of keys (the second warpgroup has none), a partial second block, odd and even numbers of
# blocks, a partial last block of the first warpgroup, the longest sequence.
@pytest.mark.parametrize("seq", [8, 64, 72, 128, 136, 200, 320, 512])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_attention_key_blocks(gpx, oracle, seq, dtype):
    ex, taps, _ = _bert(gpx, oracle, 3, seq, dtype)
    for layer in (0, 1):
        name = f"encoder.layer.{layer}.attention.context"
        assert _rel(ex.model.get(name).reshape(taps[name].shape), taps[name]) <= TOL[dtype], name
    ex.clear()


# Two rows a warp from 9472 rows on a 148-SM device: below, at a multiple of the 16-row tile, and with half a
# tile left over.
@pytest.mark.parametrize("batch,seq", [(74, 120), (80, 120), (79, 120)])
def test_layernorm_rows_per_tile(gpx, oracle, batch, seq):
    ex, taps, heads = _bert(gpx, oracle, batch, seq, "float32")
    name = "encoder.layer.0.output"
    assert _rel(ex.model.get(name).reshape(taps[name].shape), taps[name]) <= TOL["float32"]
    assert _rel(ex.get_output("heads"), heads) <= TOL["float32"]
    ex.clear()


@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_projections_share_one_product_and_keep_their_tensors(gpx, oracle, dtype):
    """Query, key and value weights are slices of one matrix: each is read and written by its own name."""
    ex, taps, heads = _bert(gpx, oracle, 2, 40, dtype)
    p = "encoder.layer.0.attention.self."
    x = taps["embeddings"].astype(np.float64)
    for part in ("query", "key", "value"):
        w, b = ex.model.get(p + part + ".weight"), ex.model.get(p + part + ".bias")
        want = x @ w.reshape(w.shape[0], -1).astype(np.float64).T + b
        assert _rel(ex.model.get(p + part + ".out").reshape(want.shape), want) <= TOL[dtype], part
    before = {part: ex.model.get(p + part + ".weight") for part in ("query", "key", "value")}
    ex.model.set(p + "key.weight", before["key"] * 2)
    for part in ("query", "key", "value"):
        assert np.array_equal(ex.model.get(p + part + ".weight"), before[part] * (2 if part == "key" else 1))
    query, value = ex.model.get(p + "query.out"), ex.model.get(p + "value.out")
    ex.execute()
    assert np.array_equal(ex.model.get(p + "query.out"), query) and np.array_equal(ex.model.get(p + "value.out"), value)
    assert not np.array_equal(ex.get_output("heads"), heads.astype(np.float32))
    ex.clear()


@pytest.mark.parametrize("batch,dtype", [(1, "float16"), (5, "float32")])
def test_batch_norm_in_the_operand(gpx, oracle, batch, dtype):
    """The normalised copy exists only in shared memory: reading it computes it, and what is written to it is
    read back, in the storage format, until the model runs."""
    ex = gpx.BaseExecutor()
    ex.init("densenet_tiny", batch=batch, seed=1, dtype=dtype)
    data = _images(gpx, batch)
    ex.set_input("data", data)
    ex.execute()
    assert ex.error() == (0, 0)
    taps = {}
    heads = oracle.forward("densenet_tiny", ex.model.params(), data, taps=taps)
    norms = [n for n in taps if ".norm" in n]
    assert norms
    for n in norms + [n for n in taps if n.endswith(".conv1") or n.endswith(".conv")]:
        assert _rel(ex.model.get(n).reshape(taps[n].shape), taps[n]) <= TOL[dtype], n
    first = ex.get_output("heads")
    assert _rel(first, heads) <= TOL[dtype]
    formed = ex.model.get(norms[0])
    ex.model.set(norms[0], formed * 2)
    assert np.array_equal(ex.model.get(norms[0]), formed * 2) and np.array_equal(ex.get_output("heads"), first)
    ex.execute()
    assert np.array_equal(ex.model.get(norms[0]), formed) and np.array_equal(ex.get_output("heads"), first)
    ex.clear()


# 2048 inputs: five rows are the most the short form keeps in shared memory.
@pytest.mark.parametrize("model,batch", [("resnet_tiny", 5), ("resnet_tiny", 6), ("resnet_tiny", 8), ("mobilenet_v2", 4)])
@pytest.mark.parametrize("dtype", ["float32", "float16"])
def test_classifier_rows_and_large_depthwise_layers(gpx, oracle, model, batch, dtype):
    """(At four images the first depthwise layers exceed four tiles an SM.)"""
    ex = gpx.BaseExecutor()
    ex.init(model, batch=batch, seed=3, dtype=dtype)
    data = _images(gpx, batch, 2)
    ex.set_input("data", data)
    ex.execute()
    assert ex.error() == (0, 0)
    taps = {}
    heads = oracle.forward(model, ex.model.params(), data, taps=taps)
    for name in [n for n in taps if n.endswith(".dw") or n == "features.0"]:
        assert _rel(ex.model.get(name).reshape(taps[name].shape), taps[name]) <= TOL[dtype], name
    assert _rel(ex.get_output("heads"), heads) <= TOL[dtype]
    ex.clear()


def test_wide_tiles_agree_with_narrow_ones(gpx):
    """80 images give the deep 3x3 layers 256-column tiles, eight images narrower ones; the sums are the same."""
    data = _images(gpx, 80, 5)
    heads = {}
    for batch in (80, 8):
        ex = gpx.BaseExecutor()
        ex.init("resnet_tiny", batch=batch, seed=3, dtype="float16")
        ex.set_input("data", data[:batch])
        ex.execute()
        assert ex.error() == (0, 0)
        heads[batch] = ex.get_output("heads")
        ex.clear()
    assert _rel(heads[80][:8], heads[8]) <= 2e-3


# Average in-degree around 200, 100, 50 and 16: eight, four, two and one id a lane (in the tiles asked for; by
# themselves graphs this small stay lists); the last graph's neighbours lie too far apart for a window.
@pytest.mark.parametrize("tile", [64, 8, 256, None])
@pytest.mark.parametrize("vertices,degree,band", [(3001, 200, 1500), (2999, 100, 900), (4000, 50, 600), (65, 16, 60), (40001, 20, 39000)])
def test_pagerank_list_forms(gpx, tmp_path, monkeypatch, vertices, degree, band, tile):
    from oracle import graphs

    if tile:
        monkeypatch.setenv("GPX_GRAPH_TILE", str(tile))

    graphs.build()
    prefix = str(tmp_path / "g" / "g.bel")
    rng = np.random.default_rng(vertices)
    rows = []
    for v in range(vertices):
        deg = int(rng.integers(0, 2 * degree))  # (vertices without edges among them)
        rows.append(np.unique(rng.integers(max(0, v - band), min(vertices, v + band + 1), deg)))
    offsets = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    neighbours = np.concatenate(rows).astype(np.uint64)
    graph_files.write_bel(prefix, offsets, neighbours, np.ones(len(neighbours), np.uint32))
    want = graphs.pagerank(offsets, neighbours)[0].astype(np.float64)
    for kind in ("base", "blp"):
        ex = gpx.BaseExecutor() if kind == "base" else gpx.BLPExecutor()
        ex.set_graph_path(prefix)
        ex.init("pagerank")
        if kind == "blp":
            word = gpx.PreemptWord(1)
            ex.set_word(word)
        ex.execute()
        err = np.abs(ex.model.get("value").astype(np.float64) - want)
        assert err.max() <= 1.1e-3 and err.mean() <= 1e-5, kind
        ex.clear()


def test_short_preemptible_forward_follows_word_and_stream(gpx):
    """execute keeps a graph of a short forward: another word, stream or trace setting has to show in it."""
    ex = gpx.BLPExecutor()
    ex.init("resnet_tiny", batch=1, seed=3)
    ex.set_input("data", _images(gpx, 1))
    words = [gpx.PreemptWord(1), gpx.PreemptWord(1)]
    streams = [gpx.Stream(1), gpx.Stream(0)]
    ex.set_word(words[0])
    ex.execute()
    want = ex.get_output("heads")
    for word in words:
        ex.set_word(word)
        for s in streams:
            word.raise_()
            ex.execute(s)
            s.sync()
            word.clear()
            assert ex.resume(s) == 0  # nothing had run
            s.sync()
            assert ex.resume(s) == -1 and np.array_equal(ex.get_output("heads"), want)
            ex.execute(s)
            assert ex.resume(s) == -1 and np.array_equal(ex.get_output("heads"), want)
    ex.clear()
    for o in words + streams:
        o.destroy()


def test_resets_are_ordered_before_later_launches(gpx, oracle):
    """A context's reset is not waited for: launches on any stream and copies still come behind it."""
    n = 300_001
    x, y = gpx.synth_uniform(n, 4, 0), gpx.synth_uniform(n, 4, 1)
    dx, dy = gpx.DeviceBuffer.from_numpy(x), gpx.DeviceBuffer.from_numpy(y)
    word = gpx.PreemptWord(1)
    ctx = gpx.BlpContext(word, kernel_id=2)
    streams = [gpx.Stream(1), gpx.Stream(0)]
    want = y
    for i in range(40):
        s = streams[i % 2]
        ctx.reset()
        gpx.axpy(0.5, dx, dy, n, ctx, s)
        s.sync()
        want = oracle.axpy(0.5, x, want)
    st = ctx.read()
    assert st["stop_index"] == -1 and st["tiles_run"] == gpx.axpy_tiles(n)
    assert np.array_equal(dy.download(np.float32, n).view(np.uint32), want.view(np.uint32))
    for o in (dx, dy, ctx, word, *streams):
        (o.free if hasattr(o, "free") else o.destroy)()


@pytest.mark.parametrize("model,seq,dtype", [("resnet50", 0, "float32"), ("mobilenet_v2", 0, "bfloat16"), ("bert_base", 128, "float16")])
def test_cluster_reduction_back_to_back(gpx, model, seq, dtype):
    """Batch-1 forwards queued behind one another: a CTA of a cluster may leave only when its partial sums have
    reached their owners, because the kernel behind it fills the shared memory it leaves.  The preemptible
    executor reduces through memory and has the same sums in the same order."""
    data = np.random.default_rng(4).integers(0, 30522, (1, seq)).astype(np.int64) if seq else _images(gpx, 1, 4)
    blp = gpx.BLPExecutor()
    blp.init(model, batch=1, seed=3, seq_len=seq, dtype=dtype)
    word, s = gpx.PreemptWord(1), gpx.Stream(0)
    blp.set_word(word)
    blp.set_input("data", data)
    blp.execute(s)
    s.sync()
    want = blp.get_output("heads")
    ex = gpx.BaseExecutor()
    ex.init(model, batch=1, seed=3, seq_len=seq, dtype=dtype)
    ex.set_input("data", data)
    for _ in range(20):
        for _ in range(20):
            ex.execute(s)
        s.sync()
        assert ex.error() == (0, 0) and np.array_equal(ex.get_output("heads"), want)
    ex.clear(), blp.clear(), word.destroy(), s.destroy()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_launch_behind_a_reset_can_be_captured(gpx, oracle, mode):
    """A launch with a context goes into a CUDA graph: the reset before it is not part of the graph, so a
    replay needs a reset of its own, and a replay without one finds every tile done."""
    import ctypes

    import torch

    n = 100_003
    x, y = gpx.synth_uniform(n, 4, 0), gpx.synth_uniform(n, 4, 1)
    dx, dy = gpx.DeviceBuffer.from_numpy(x), gpx.DeviceBuffer.from_numpy(y)
    word = gpx.PreemptWord(1)
    ctx = gpx.BlpContext(word, kernel_id=2)
    m, nn, k = 256, 512, 128
    a = oracle.f32_to_bf16(gpx.synth_uniform(m * k, 3, 0).reshape(m, k))
    b = oracle.f32_to_bf16(gpx.synth_uniform(nn * k, 3, 1).reshape(nn, k))
    da, db, dc = gpx.DeviceBuffer.from_numpy(a), gpx.DeviceBuffer.from_numpy(b), gpx.DeviceBuffer(m * nn * 2)
    gctx, gblp = gpx.GemmContext(), gpx.BlpContext(word, kernel_id=3)
    gctx.reset()
    stream = torch.cuda.Stream()
    handle = ctypes.c_void_p(stream.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    ctx.reset()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        gpx.axpy(0.5, dx, dy, n, ctx, handle)
        gpx.gemm_bf16(da, db, dc, m, nn, k, gctx, gblp, handle)
    assert np.array_equal(dy.download(np.float32, n), y)  # captured, not run
    want = y
    for fresh in (True, False, True):
        if fresh and want is not y:
            ctx.reset(), gctx.reset(), gblp.reset()
            gpx.device_sync()
        with torch.cuda.stream(stream):
            graph.replay()
        stream.synchronize()
        want = oracle.axpy(0.5, x, want) if fresh else want
        assert np.array_equal(dy.download(np.float32, n).view(np.uint32), want.view(np.uint32))
    assert gctx.status() == (0, 0)
    got = oracle.bf16_to_f32(dc.download(np.uint16, m * nn)).reshape(m, nn).astype(np.float64)
    exact = oracle.gemm_bf16_nt(a, b)
    assert np.all(np.abs(got - exact) <= np.abs(exact) * 2.0 ** -8 + np.abs(exact).max() * 1e-5)
    del graph
    for o in (dx, dy, da, db, dc, ctx, gctx, gblp, word):
        (o.free if hasattr(o, "free") else o.destroy)()


def test_context_addresses_and_new_streams_come_behind_a_reset(gpx, oracle):
    """The raw launch argument is handed out only when the reset is through, and a stream that reuses the handle
    of a destroyed one is ordered like any other."""
    import ctypes

    from gpreempt_b200 import binding as B

    n = 100_003
    x, y = gpx.synth_uniform(n, 4, 0), gpx.synth_uniform(n, 4, 1)
    dx, dy = gpx.DeviceBuffer.from_numpy(x), gpx.DeviceBuffer.from_numpy(y)
    word = gpx.PreemptWord(1)
    ctx = gpx.BlpContext(word, kernel_id=2)
    want = y
    for i in range(20):
        s = gpx.Stream(1)
        ctx.reset()
        if i % 2:
            gpx.axpy(0.5, dx, dy, n, ctx, s)
        else:
            arg = ctx.struct()
            assert not ctx._pending
            B.check(B.load().gpx_axpy_f32(0.5, dx.ptr, dy.ptr, n, 0, ctypes.byref(arg), s.handle))
        s.sync()
        s.destroy()
        want = oracle.axpy(0.5, x, want)
        assert ctx.read()["tiles_run"] == gpx.axpy_tiles(n)
    assert np.array_equal(dy.download(np.float32, n).view(np.uint32), want.view(np.uint32))
    for o in (dx, dy, ctx, word):
        (o.free if hasattr(o, "free") else o.destroy)()


@pytest.mark.parametrize("model", ["bert_tiny", "densenet_tiny"])
def test_every_tensor_and_function_has_its_own_name(gpx, tmp_path, model):
    """Tensors of fused layers are read and written under their names, the fused ones' too, and an exported
    directory lists a kernel for every function."""
    import json

    ex = gpx.BaseExecutor()
    ex.init(model, batch=2, seed=7, seq_len=16 if model == "bert_tiny" else 0)
    data = np.random.default_rng(1).integers(0, 1000, (2, 16)).astype(np.int64) if model == "bert_tiny" else _images(gpx, 2)
    ex.set_input("data", data)
    ex.execute()
    heads = ex.get_output("heads")
    infos = [ex.model.get_storage_info(i) for i in range(ex.model.get_storage_num())]
    values = {i["name"]: ex.model.get(i["name"]) for i in infos if i["stype"] == "float32" and i["name"] != "data"}
    for name, v in values.items():
        ex.model.set(name, v)
        assert np.array_equal(ex.model.get(name), v), name
    for name, v in values.items():
        if name.endswith(".qkv.weight"):
            parts = [values[name.replace(".query.out.qkv", "." + part)] for part in ("query", "key", "value")]
            assert np.array_equal(v, np.concatenate(parts))
    ex.execute()
    assert np.array_equal(ex.get_output("heads"), heads)
    ex.model.export_dir(str(tmp_path / model))
    host = json.load(open(tmp_path / model / "host.json"))
    assert all(f["kernels"] for f in host["funcs"])
    ex.clear()


@pytest.mark.parametrize("channels", [752, 768, 784])
def test_depthwise_filter_beside_the_kernels_own_shared_memory(gpx, tmp_path, channels):
    """A 4x4 filter of 768 channels is the whole of the default 48 KB: it does not go to shared memory."""
    import ctypes
    import json

    import torch

    from gpreempt_b200 import binding as B

    def param(name):
        return {"op": "null", "name": name, "inputs": [], "attrs": {"gpx_kind": "param", "init_std": 0.1, "init_mean": 0.0}}

    def layer(name, fn, inputs, kernel, stride, pad):
        return {"op": "tvm_op", "name": name, "inputs": [[i, 0, 0] for i in inputs],
                "attrs": {"func_name": fn, "kernel": kernel, "stride": stride, "padding": pad, "activation": 0}}

    n, hw = 2, 9
    nodes = [{"op": "null", "name": "data", "inputs": [], "attrs": {"gpx_kind": "input"}},
             param("a.weight"), param("a.bias"), layer("a", "gpx_conv2d", [0, 1, 2], 1, 1, 0),
             param("b.weight"), param("b.bias"), layer("b", "gpx_depthwise_conv2d", [3, 4, 5], 4, 1, 1),
             layer("pool", "gpx_avg_pool2d", [6], hw - 1, 1, 0),
             param("heads.weight"), param("heads.bias"), layer("heads", "gpx_conv2d", [7, 8, 9], 1, 1, 0)]
    shapes = [[n, 3, hw, hw], [channels, 3, 1, 1], [channels], [n, channels, hw, hw], [channels, 1, 4, 4], [channels],
              [n, channels, hw - 1, hw - 1], [n, channels, 1, 1], [1000, channels, 1, 1], [1000], [n, 1000]]
    graph = {"nodes": nodes, "heads": [[10, 0, 0]], "gpx": {"model": "dw4", "batch": n, "dtype": "float32", "pad_channels": False},
             "attrs": {"dltype": ["list_str", ["float32"] * len(nodes)], "shape": ["list_shape", shapes]}}
    (tmp_path / "mod.json").write_text(json.dumps(graph))
    (tmp_path / "host.json").write_text(json.dumps(
        {"temp_args": [], "funcs": [{"name": x["attrs"]["func_name"], "kernels": [{}]} for x in nodes if x["inputs"]]}))
    ex = gpx.BaseExecutor()
    ex.model = gpx.Model(str(tmp_path))
    B.check(B.load().gpx_exec_create(ex.model.handle, B.EXEC_BASE, ctypes.byref(ex.handle)))
    ex.model.init_random(5)
    x = gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw)
    ex.set_input("data", x)
    ex.execute()
    assert ex.error() == (0, 0)
    p = {k: torch.from_numpy(v).double() for k, v in ex.model.params().items()}
    a = torch.nn.functional.conv2d(torch.from_numpy(x).double(), p["a.weight"], p["a.bias"])
    want = torch.nn.functional.conv2d(a, p["b.weight"], p["b.bias"], padding=1, groups=channels).numpy()
    assert _rel(ex.model.get("b"), want) <= TOL["float32"]
    ex.clear()


def test_short_forward_is_made_a_graph_only_when_it_repeats(gpx):
    """Setting the word makes nothing, a run after the graph of one's own was captured uses that, and runs that
    alternate between settings go kernel by kernel; all end with the same bits."""
    import time

    word = gpx.PreemptWord(1)
    streams = [gpx.Stream(1), gpx.Stream(0)]
    outs, host = [], {}
    for use in ("alternating", "repeating", "captured"):
        ex = gpx.BLPExecutor()
        ex.init("resnet_tiny", batch=1, seed=3)
        ex.set_input("data", _images(gpx, 1))
        ex.set_word(word)
        if use == "captured":
            ex.capture_graph(streams[0])
        for i in range(12):
            s = streams[i % 2 if use == "alternating" else 0]
            s.sync()
            t0 = time.perf_counter()
            ex.execute(s)
            host.setdefault(use, []).append(time.perf_counter() - t0)
            s.sync()
            outs.append(ex.get_output("heads"))
            assert ex.getStopPoint(s) == -1
        ex.clear()
    assert all(np.array_equal(o, outs[0]) for o in outs)
    # 33 launches against one: the host time of the last runs tells which way they went
    assert np.median(host["repeating"][4:]) < 0.5 * np.median(host["alternating"][4:])
    for o in [word] + streams:
        o.destroy()


def _pagerank(gpx, tmp_path, rows, prefix_name="g"):
    """The graph in files, its kernels' edge-pass tiles, and one run against the oracle."""
    from oracle import graphs

    graphs.build()
    prefix = str(tmp_path / prefix_name / "g.bel")
    offsets = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    neighbours = np.concatenate(rows).astype(np.uint64)
    graph_files.write_bel(prefix, offsets, neighbours, None)
    ex = gpx.BaseExecutor()
    ex.set_graph_path(prefix)
    ex.init("pagerank")
    tiles = {i["total_tiles"] for i in (ex.model.get_kernel_info(k) for k in range(ex.get_kernel_num())) if ".edges." in i["name"]}
    ex.execute()
    err = np.abs(ex.model.get("value").astype(np.float64) - graphs.pagerank(offsets, neighbours)[0].astype(np.float64))
    assert err.max() <= 1.1e-3 and err.mean() <= 1e-5
    ex.clear()
    assert len(tiles) == 1
    return tiles.pop()


@pytest.mark.parametrize("vertices", [12223, 12224, 12287, 12288])
def test_pagerank_longest_window(gpx, tmp_path, vertices):
    """Every tile reads the first and the last vertex, so its window is the whole graph: up to 12 223 deltas go to
    shared memory beside the kernel's own variables, more stay in lists (tiles of 16 vertices)."""
    rng = np.random.default_rng(vertices)
    rows = [np.unique(rng.integers(0, vertices, 400)) for _ in range(vertices)]
    rows[0] = rows[-1] = np.arange(vertices)
    lists = _pagerank(gpx, tmp_path, rows) == -(-vertices // 16)
    assert lists == (vertices > 12223)


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_attention_rows_that_one_key_dominates(gpx, dtype):
    """With scores spread wide a row of the context is nearly one row of the values, so its only error is the
    rounding of the result, the probability of the dominating key being exactly 1.  From the stored queries,
    keys and values, in 64 bits."""
    import torch

    ex = gpx.BaseExecutor()
    ex.init("bert_tiny", batch=16, seed=1, seq_len=512, dtype=dtype)
    name = "encoder.layer.0.attention."
    ex.model.set(name + "self.query.weight", ex.model.get(name + "self.query.weight") * 192)
    ex.set_input("data", np.random.default_rng(1).integers(0, 1000, (16, 512)).astype(np.int64))
    ex.execute()
    assert ex.error() == (0, 0)
    q, k, v = (torch.from_numpy(ex.model.get(name + "self." + part + ".out")).double() for part in ("query", "key", "value"))
    got = torch.from_numpy(ex.model.get(name + "context")).double()
    batch, seq, width = q.shape
    q, k, v = (t.reshape(batch, seq, width // 64, 64).transpose(1, 2) for t in (q, k, v))
    want = (torch.softmax(q @ k.transpose(-1, -2) / 8.0, -1) @ v).transpose(1, 2).reshape(batch, seq, width)
    rounded = want.to(torch.float16 if dtype == "float16" else torch.bfloat16).double()
    error, rounding = (float((t - want).norm() / want.norm()) for t in (got, rounded))
    assert error <= 1.03 * rounding, (error, rounding)
    ex.clear()


@pytest.mark.parametrize("value", [0.9, -2.0, np.inf, np.nan, 3e20])
def test_miniweather_tiles_that_divide(gpx, value):
    """One density beyond what the quotients by reciprocals take makes its tile divide: every cell its stencil does
    not reach keeps its bits, along x and along z."""
    ex = gpx.BaseExecutor()
    ex.init("miniweather_320x160")
    state = ex.model.get("state").copy()
    rng = np.random.default_rng(3)
    state[:, 2:-2, 2:-2] += rng.normal(0, [[[1e-3]], [[1]], [[1]], [[0.3]]], (4, 160, 320)).astype(np.float32)
    row, col = 70, 150
    outs = {}
    for wild in (False, True):
        for kernel in (0, 3):  # the first stage along x, the first along z
            s = state.copy()
            if wild:
                s[0, row, col] = value
            for name in ("state", "state_tmp", "state_tmp2"):
                ex.model.set(name, s)
            ex.launch_kernel(kernel)
            outs[wild, kernel] = ex.model.get("state_tmp")[:, 2:-2, 2:-2]
    r, c = row - 2, col - 2
    for kernel in (0, 3):
        a, b = outs[False, kernel], outs[True, kernel]
        assert np.all(np.isfinite(a))
        near = np.zeros(a.shape[1:], bool)
        if kernel == 0:
            near[r, c - 3:c + 4] = True
        else:
            near[r - 3:r + 4, c] = True
        assert np.array_equal(a[:, ~near].view(np.uint32), b[:, ~near].view(np.uint32)), kernel
        assert not np.array_equal(a[:, near], b[:, near])
    ex.clear()


def _sym(vertices, a, b):
    """Rows of the symmetric graph with these edges and a chain through all vertices."""
    chain = np.arange(vertices - 1)
    a, b = np.concatenate([a, chain]), np.concatenate([b, chain + 1])
    key = np.unique(np.concatenate([a * vertices + b, b * vertices + a]))
    return np.split(key % vertices, np.cumsum(np.bincount(key // vertices, minlength=vertices))[:-1])


def _banded(rng, vertices, degree, band):
    a = np.repeat(np.arange(vertices), degree // 2)
    b = a + rng.integers(1, band + 1, len(a)) * (rng.integers(0, 2, len(a)) * 2 - 1)
    inside = (b >= 0) & (b < vertices)
    return _sym(vertices, a[inside], b[inside])


def test_pagerank_form_follows_the_graph(gpx, tmp_path, monkeypatch):
    """Packed tiles of 64 or 32 vertices where there are enough of them, lists (tiles of 16) for small graphs, for
    neighbours without locality and for skewed degrees; GPX_GRAPH_TILE sets the tile of either form."""
    rng = np.random.default_rng(5)
    sm = gpx.device_info()["sm_count"]
    large, middle, small = 256 * sm + 37, 128 * sm + 5, 60 * sm + 3
    band = _banded(rng, large, 20, 300)
    assert _pagerank(gpx, tmp_path, band, "a") == -(-large // 64)
    assert _pagerank(gpx, tmp_path, _banded(rng, middle, 20, 200), "b") == -(-middle // 32)
    assert _pagerank(gpx, tmp_path, _banded(rng, small, 60, 300), "c") == -(-small // 16)
    n = min(12000, middle // 32 * 32)
    assert _pagerank(gpx, tmp_path, _sym(n, rng.integers(0, n, 10 * n), rng.integers(0, n, 10 * n)), "d") == -(-n // 16)
    hubs = (large * rng.random(8 * large) ** 4).astype(int)
    near = np.clip(hubs + rng.integers(-1500, 1501, len(hubs)), 0, large - 1)
    assert _pagerank(gpx, tmp_path, _sym(large, hubs, near), "e") == -(-large // 16)
    for tile in (16, 40, 128):
        monkeypatch.setenv("GPX_GRAPH_TILE", str(tile))
        assert _pagerank(gpx, tmp_path, band, "f%d" % tile) == -(-large // tile)


def test_launches_follow_the_current_context(gpx):
    """The handle of a kernel belongs to a context, and a thread may change its own: a model made and run in a second
    context of the device gives the bits of one in the first, before, between and after."""
    import ctypes

    driver = ctypes.CDLL("libcuda.so.1")

    def run():
        ex = gpx.BaseExecutor()
        ex.init("miniweather_200x104")
        ex.execute()
        state = ex.model.get("state")
        ex.clear()
        return state

    want = run()
    for _ in range(2):
        ctx = ctypes.c_void_p()
        assert driver.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0) == 0  # (and makes it current)
        try:
            assert np.array_equal(run(), want)
        finally:
            driver.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p()))
            driver.cuCtxDestroy_v2(ctx)
        assert np.array_equal(run(), want)
