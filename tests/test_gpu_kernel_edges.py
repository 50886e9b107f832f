"""Small graphs at the sizes where a layer's kernel meets a tile's edge, a remainder or the line of a rule that picks
between two kernels.  Every value is compared with 64-bit arithmetic on the operands that the layer itself read, so the
bounds are the rounding of the stored result plus that of 32-bit sums."""
import ctypes
import json
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Half a unit in the last place of the stored type (two bf16 planes hold 16 bits and more, but a sum of products of them
# drops the product of the low planes: 2^-16 an operand), of a value itself; and what 32-bit sums of a few thousand terms
# and the two roundings of an intermediate add, of the tensor's largest value.
HALF_ULP = {"float32": 2.0 ** -15, "float16": 2.0 ** -11, "bfloat16": 2.0 ** -8}
SUMS = 2e-5


def _close(got, want, dtype, what):
    got, want = got.astype(np.float64), want.astype(np.float64)
    bound = HALF_ULP[dtype] * np.abs(want) + SUMS * np.max(np.abs(want))
    worst = np.max(np.abs(got - want) / bound)
    assert worst <= 1, f"{what}: {worst:.2f} times the bound"


def _param(name, std=0.1, kind="param"):
    return {"op": "null", "name": name, "inputs": [], "attrs": {"gpx_kind": kind, "init_std": std, "init_mean": 0.0}}


class _Graph:
    """A graph as an exported model directory holds it."""

    def __init__(self, batch, dtype, pad_channels=False):
        self.batch, self.dtype, self.pad_channels = batch, dtype, pad_channels
        self.nodes, self.shapes, self.types = [], [], []

    def add(self, node, shape, dltype="float32"):
        self.nodes.append(node), self.shapes.append(list(shape)), self.types.append(dltype)
        return len(self.nodes) - 1

    def input(self, *shape, ids=False):
        return self.add({"op": "null", "name": "data", "inputs": [], "attrs": {"gpx_kind": "input"}}, shape, "int64" if ids else "float32")

    def op(self, name, fn, inputs, shape, **attrs):
        return self.add({"op": "tvm_op", "name": name, "inputs": [[i, 0, 0] for i in inputs], "attrs": dict(attrs, func_name=fn)}, shape)

    def conv(self, name, src, cout, kernel=1, pad=0, act=0, residual=None, std=0.1):
        n, c, h, w = self.shapes[src]
        inputs = [src, self.add(_param(name + ".weight", std), [cout, c, kernel, kernel]), self.add(_param(name + ".bias"), [cout])]
        attrs = {"kernel": kernel, "stride": 1, "padding": pad, "activation": act}
        if residual is not None:
            inputs.append(residual)
            attrs["residual"] = True
        return self.op(name, "gpx_conv2d", inputs, [n, cout, h + 2 * pad - kernel + 1, w + 2 * pad - kernel + 1], **attrs)

    def pool(self, name, src, fn, kernel, stride, pad):
        n, c, h, w = self.shapes[src]
        return self.op(name, fn, [src], [n, c, (h + 2 * pad - kernel) // stride + 1, (w + 2 * pad - kernel) // stride + 1],
                       kernel=kernel, stride=stride, padding=pad, activation=0)

    def heads(self, src):
        """Averages over the image and a classifier: what ends every graph of images here."""
        n, c, h, w = self.shapes[src]
        assert h == w
        return self.conv("heads", self.pool("mean", src, "gpx_avg_pool2d", h, 1, 0), 16)

    def load(self, gpx, path, cls=None):
        from gpreempt_b200 import binding as B

        path.mkdir(exist_ok=True)
        graph = {"nodes": self.nodes, "heads": [[len(self.nodes) - 1, 0, 0]],
                 "gpx": {"model": "edges", "batch": self.batch, "dtype": self.dtype, "pad_channels": self.pad_channels},
                 "attrs": {"dltype": ["list_str", self.types], "shape": ["list_shape", self.shapes]}}
        (path / "mod.json").write_text(json.dumps(graph))
        (path / "host.json").write_text(json.dumps(
            {"temp_args": [], "funcs": [{"name": x["attrs"]["func_name"], "kernels": [{}]} for x in self.nodes if x["inputs"]]}))
        ex = (cls or gpx.BaseExecutor)()
        ex.model = gpx.Model(str(path))
        kind = (cls or gpx.BaseExecutor).KIND
        B.check(B.load().gpx_exec_create(ex.model.handle, kind, ctypes.byref(ex.handle)))
        ex.model.init_random(5)
        return ex


def _conv64(ex, name, src, dtype, pad=0, stride=1, groups=1, act=0, residual=None, padded=False):
    import torch

    def image(key):
        x = torch.from_numpy(ex.model.get(key)).double()
        return x.reshape(*x.shape[:2], 1, 1) if x.dim() == 2 else x

    w = torch.from_numpy(ex.model.get(name + ".weight"))
    if dtype != "float32" and groups == 1 and (padded or w.shape[1] % 64 == 0):  # (read back as the exact 32-bit copy; tensor cores multiply 16 bits)
        w = w.to(getattr(torch, dtype))
    out = torch.nn.functional.conv2d(image(src), w.double(), torch.from_numpy(ex.model.get(name + ".bias")).double(),
                                     padding=pad, stride=stride, groups=groups)
    if residual is not None:
        out = out + image(residual)
    return (torch.relu(out) if act else out).numpy().reshape(ex.model.shape(name))


# 3x3 layers of 32 and 64 output channels, from 1 024 padded rows on: a last tile of one row and of all but one, several
# blocks of input channels, one image wider than a tile, and the smallest that the rule takes (below: one block of rows less).
@pytest.mark.parametrize("cout,cin,n,hw", [(32, 64, 9, 9), (32, 128, 2, 33), (32, 128, 1, 130), (32, 64, 4, 15), (32, 64, 4, 14),
                                           (64, 64, 9, 9), (64, 64, 2, 33), (64, 64, 1, 140), (64, 64, 5, 28)])
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_narrow_3x3_layers(gpx, tmp_path, monkeypatch, cout, cin, n, hw, dtype):
    def build(path):
        g = _Graph(n, dtype)
        x = g.conv("a", g.input(n, 3, hw, hw), cin)
        x = g.conv("b", x, cout, 3, 1, act=1)
        g.heads(g.conv("c", x, cout, 3, 1) if cin == cout else x)
        ex = g.load(gpx, path)
        ex.set_input("data", gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw))
        ex.execute()
        assert ex.error() == (0, 0)
        return ex

    ex = build(tmp_path / "narrow")
    _close(ex.model.get("b"), _conv64(ex, "b", "a", dtype, pad=1, act=1), dtype, "b")
    if cin == cout:
        _close(ex.model.get("c"), _conv64(ex, "c", "b", dtype, pad=1), dtype, "c")
    monkeypatch.setenv("GPX_CONV_NARROW", "0")
    general = build(tmp_path / "general")
    a, b = ex.model.get("b"), general.model.get("b")
    assert np.array_equal(ex.model.get("a"), general.model.get("a"))
    # 32-bit sums of the same products in another order: at most one unit in the last place apart
    np.testing.assert_allclose(a, b, rtol=2 * HALF_ULP[dtype], atol=SUMS * np.abs(b).max())
    ex.clear(), general.clear()


@pytest.mark.parametrize("cout", [32, 64])
@pytest.mark.parametrize("transport", [0, 1])
def test_narrow_3x3_layers_end_with_the_same_bits_after_a_stop(gpx, tmp_path, cout, transport):
    n, hw = 24, 56
    g = _Graph(n, "float16")
    x = g.conv("in", g.input(n, 3, hw, hw), 64)
    for i in range(8):
        x = g.conv(f"n{i}", x, cout, 3, 1, act=1, std=0.06)
        if cout != 64:
            x = g.conv(f"w{i}", x, 64)
    g.heads(x)
    names = [f"n{i}" for i in range(8)]
    data = gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw)
    ex = g.load(gpx, tmp_path / "be", gpx.BLPExecutor)
    word, s = gpx.PreemptWord(transport), gpx.Stream(1)
    ex.set_word(word)
    ex.set_input("data", data)
    ex.execute(s)
    s.sync()
    want = {k: ex.model.get(k) for k in names}
    t0 = time.perf_counter()
    ex.execute(s)
    s.sync()
    run = time.perf_counter() - t0
    rng, stops = np.random.default_rng(11), 0
    for _ in range(8):
        ex.set_input("data", data * 0)
        ex.execute(s)
        s.sync()  # nothing stale can pass
        ex.set_input("data", data)
        word.clear()
        time.sleep(0.001)
        ex.execute(s)
        for turn in range(40):
            if turn < 4:
                until = time.perf_counter() + float(rng.uniform(0, run / 2))
                while time.perf_counter() < until:
                    pass
                word.raise_()
            s.sync()
            word.clear()
            time.sleep(0.0005)
            if ex.resume(s) == -1:
                break
            stops += 1
        else:
            raise AssertionError("does not end")
        s.sync()
        assert ex.error() == (0, 0)
        for k in names:
            assert np.array_equal(ex.model.get(k), want[k]), k
    assert stops > 0
    ex.clear(), word.destroy(), s.destroy()


# Latency-critical launches: one tile and no split (64 channels), splits over a cluster (512 to 2 048), rows that end inside a
# split's share or leave splits without any, output channels that end inside a block of columns, with and without a residual.
@pytest.mark.parametrize("hw", [1, 3, 5, 7, 11, 14])
@pytest.mark.parametrize("cin,cout", [(64, 64), (64, 208), (512, 80), (1024, 256), (2048, 64)])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_latency_critical_layers_of_few_rows(gpx, tmp_path, hw, cin, cout, dtype):
    g = _Graph(1, dtype)
    x = g.input(1, 3, hw, hw)
    res = g.conv("r", x, cout)
    x = g.conv("b", g.conv("a", x, cin), cout, act=1, residual=res, std=0.03)
    g.heads(g.conv("c", x, cout, std=0.03))
    ex = g.load(gpx, tmp_path / "hp")
    ex.set_input("data", gpx.synth_normal(3 * hw * hw, 2, 0).reshape(1, 3, hw, hw))
    for _ in range(3):  # (a launch finds the next one's weights under way only where there is a predecessor)
        ex.execute()
    assert ex.error() == (0, 0)
    _close(ex.model.get("b"), _conv64(ex, "b", "a", dtype, act=1, residual="r"), dtype, "b")
    _close(ex.model.get("c"), _conv64(ex, "c", "b", dtype), dtype, "c")
    ex.clear()


# The batch norm in the operand, mapped in shared memory (two planes, latency-critical launches) or into tensor memory: one
# block of channels, a last one in part, more than the ring holds; a last tile of one row and a CTA's second tile.
@pytest.mark.parametrize("cin,cout,n,hw", [(64, 128, 1, 1), (64, 64, 3, 13), (96, 128, 1, 23), (160, 128, 129, 1), (448, 128, 2, 9), (704, 64, 5, 7),
                                           (128, 128, 64, 20)])
@pytest.mark.parametrize("preemptible", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_batch_norm_in_the_operand_of_one_layer(gpx, tmp_path, cin, cout, n, hw, preemptible, dtype):
    g = _Graph(n, dtype, pad_channels=True)
    x = g.conv("a", g.input(n, 3, hw, hw), cin)
    x = g.op("norm", "gpx_affine", [x, g.add(_param("norm.weight"), [cin]), g.add(_param("norm.bias"), [cin])], g.shapes[x],
             kernel=1, stride=1, padding=0, activation=1, in_channels=cin)
    g.heads(g.conv("b", x, cout, act=1))
    ex = g.load(gpx, tmp_path / "norm", gpx.BLPExecutor if preemptible else gpx.BaseExecutor)
    rng, s = np.random.default_rng(cin), gpx.Stream(1)
    ex.model.set("norm.weight", rng.normal(1, 0.3, cin).astype(np.float32))
    ex.model.set("norm.bias", rng.normal(0, 0.3, cin).astype(np.float32))
    if preemptible:
        word = gpx.PreemptWord(1)
        ex.set_word(word)
    ex.set_input("data", gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw))
    ex.execute(s)
    s.sync()
    assert ex.error() == (0, 0)
    _close(ex.model.get("b"), _conv64(ex, "b", "norm", dtype, act=1, padded=True), dtype, "b")
    ex.clear(), s.destroy()
    if preemptible:
        word.destroy()


# One to four vectors a lane, partial ones, and rows on both sides of 32 an SM (the last row of a tile alone).
@pytest.mark.parametrize("width", [8, 256, 264, 512, 520, 768, 776, 1024])
@pytest.mark.parametrize("batch,seq", [(1, 2), (3, 7), (593, 8)])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_layernorm_widths(gpx, tmp_path, width, batch, seq, dtype):
    g = _Graph(batch, dtype)
    ids = g.input(batch, seq, ids=True)
    word, pos = (g.add(_param(k, 1.0, "table"), s) for k, s in (("word", [50, width]), ("pos", [64, width])))
    w, b = (g.add(_param("emb." + k), [width]) for k in ("weight", "bias"))
    x = g.op("emb", "gpx_layer_norm", [ids, word, pos, w, b], [batch, seq, width])
    w, b = (g.add(_param("ln." + k), [width]) for k in ("weight", "bias"))
    x = g.op("ln", "gpx_layer_norm", [x, w, b], [batch, seq, width])
    w, b = (g.add(_param("heads." + k), [width]) for k in ("weight", "bias"))
    g.op("heads", "gpx_layer_norm", [x, w, b], [batch, seq, width])
    ex = g.load(gpx, tmp_path / "ln")
    rng = np.random.default_rng(width)
    for name in ("emb", "ln", "heads"):
        ex.model.set(name + ".weight", rng.normal(1, 0.1, width).astype(np.float32))
        ex.model.set(name + ".bias", rng.normal(0, 0.1, width).astype(np.float32))
    data = rng.integers(0, 50, (batch, seq)).astype(np.int64)
    ex.set_input("data", data)
    ex.execute()
    assert ex.error() == (0, 0)

    def norm(x, name):
        x = x.astype(np.float64)
        c = x - x.mean(-1, keepdims=True)
        y = c / np.sqrt((c * c).mean(-1, keepdims=True) + 1e-12)
        return y * ex.model.get(name + ".weight").reshape(-1) + ex.model.get(name + ".bias").reshape(-1)

    def stored(name):
        return ex.model.get(name).reshape(batch, seq, width)

    table = ex.model.get("word").reshape(50, width).astype(np.float64)[data] + ex.model.get("pos").reshape(64, width)[None, :seq]
    _close(stored("emb"), norm(table, "emb"), dtype, "emb")
    _close(stored("ln"), norm(stored("emb"), "ln"), dtype, "ln")
    _close(ex.get_output("heads").reshape(batch, seq, width), norm(stored("ln"), "heads"), "float32", "heads")
    ex.clear()


# Strips of four (stride 1) or two pixels where the rows end inside one, channels that do not fill a block of 64, both
# sides of four vectors a thread.
@pytest.mark.parametrize("channels,n,hw", [(40, 10, 57), (40, 9, 57), (8, 40, 63), (96, 13, 37), (144, 2, 13), (24, 1, 1)])
@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_depthwise_strips(gpx, tmp_path, channels, n, hw, stride, dtype):
    g = _Graph(n, dtype)
    x = g.conv("a", g.input(n, 3, hw, hw), channels)
    out = (hw - 1) // stride + 1
    x = g.op("b", "gpx_depthwise_conv2d", [x, g.add(_param("b.weight", 0.3), [channels, 1, 3, 3]), g.add(_param("b.bias"), [channels])],
             [n, channels, out, out], kernel=3, stride=stride, padding=1, activation=1)
    g.heads(g.conv("c", x, 32))
    ex = g.load(gpx, tmp_path / "dw")
    ex.set_input("data", gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw))
    ex.execute()
    assert ex.error() == (0, 0)
    _close(ex.model.get("b"), _conv64(ex, "b", "a", dtype, pad=1, stride=stride, groups=channels, act=1), dtype, "b")
    _close(ex.model.get("c"), _conv64(ex, "c", "b", dtype), dtype, "c")  # (the channels that fill its block are read as zeros)
    ex.clear()


# A warp to a query up to 48 keys, up to 64 where there are few tiles: one key, the lanes' remainders, both sides of both lines.
@pytest.mark.parametrize("batch,seq", [(1, 1), (2, 2), (3, 5), (2, 31), (2, 32), (2, 33), (3, 47), (200, 48), (2, 49), (2, 63), (2, 64), (200, 64), (2, 65)])
def test_attention_over_few_keys(gpx, batch, seq):
    import torch

    from gpreempt_b200 import binding as B

    ex = gpx.BaseExecutor()
    ex.init("distilbert_tiny", batch=batch, seed=3, seq_len=seq)
    ex.set_input("data", np.random.default_rng(seq).integers(0, 1000, (batch, seq)).astype(np.int64))
    ex.execute()
    assert ex.error() == (0, 0)
    prefix = "transformer.layer.0.attention."

    def tokens(name):  # (by its bytes: the shape of a sequence of one has no token axis)
        out = np.empty((batch, seq, 128), np.float32)
        B.check(B.load().gpx_model_get(ex.model.handle, (prefix + name).encode(), out.ctypes.data_as(ctypes.c_void_p), out.nbytes, None))
        gpx.device_sync()
        return out

    q, k, v = (torch.from_numpy(tokens(p + "_lin.out")).double().reshape(batch, seq, 2, 64).transpose(1, 2) for p in "qkv")
    want = (torch.softmax(q @ k.transpose(-1, -2) / 8.0, -1) @ v).transpose(1, 2).reshape(batch, seq, 128).numpy()
    _close(tokens("context"), want, "float32", "context")
    ex.clear()


# Both windows with an instance of their own, odd images, padding at all edges, tiles that end inside one vector's row, and
# values a maximum has to get right: whole windows of minus infinity.
@pytest.mark.parametrize("fn,kernel,stride,pad", [("max", 3, 2, 1), ("max", 3, 1, 1), ("max", 3, 2, 0), ("max", 2, 2, 0), ("avg", 2, 2, 0), ("max", 2, 1, 1)])
@pytest.mark.parametrize("n,channels,hw", [(1, 8, 3), (3, 40, 17), (7, 64, 57)])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_pool_windows(gpx, tmp_path, fn, kernel, stride, pad, n, channels, hw, dtype):
    import torch

    g = _Graph(n, dtype)
    x = g.conv("a", g.input(n, 3, hw, hw), channels)
    x = g.pool("p", x, f"gpx_{fn}_pool2d", kernel, stride, pad)
    g.heads(x)
    ex = g.load(gpx, tmp_path / "pool")
    ex.set_input("data", gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw))
    ex.execute()
    assert ex.error() == (0, 0)
    kernels = [ex.model.get_kernel_info(i)["name"] for i in range(ex.get_kernel_num())]
    if fn == "max" and dtype != "float32":  # (infinity split into two planes is not a number)
        a = ex.model.get("a").copy()
        a[0, :, 0, 0], a[0, :, 1, 1], a[-1, 0] = -np.inf, 0.0, -np.inf
        ex.model.set("a", a)
        ex.launch_kernel(kernels.index("p"))
    a = torch.from_numpy(ex.model.get("a")).double()
    want = (torch.nn.functional.max_pool2d(a, kernel, stride, pad) if fn == "max" else torch.nn.functional.avg_pool2d(a, kernel, stride, pad)).numpy()
    got = ex.model.get("p").astype(np.float64).reshape(want.shape)
    if fn == "max":
        assert np.array_equal(got, want)
    else:
        _close(got, want, dtype, "p")
    ex.clear()


# Rows of four, two and one cells a lane, last segments of 61 to 124 cells and a last tile of one segment; along z heights
# that do not divide.
@pytest.mark.parametrize("nx,nz", [(500, 20), (124, 10), (126, 33), (125, 17), (249, 20), (373, 9), (1026, 30)])
def test_miniweather_remainders(gpx, nx, nz):
    from oracle import miniweather as mw

    mw.build()
    ex = gpx.BaseExecutor()
    ex.init(f"miniweather_{nx}x{nz}")
    orc = mw.Oracle(nx, nz)
    for step in (1, 2):
        ex.execute()
        orc.timestep()
        got, want = ex.model.get("state"), orc.state
        # (bounds a time step: the pressure's last place in a flux of 1e5 Pa, scaled by dt/dx; see test_gpu_miniweather)
        for v, bound in enumerate((2e-6, 6e-4, 6e-4, 2e-4)):
            assert np.max(np.abs(mw.interior(got)[v].astype(np.float64) - mw.interior(want)[v])) <= bound * step, (step, v)
    ex.clear()


# Widths of 124 k + 1 cells from 3 721 on: the last segment of a row has a single cell, so the one before it reads a cell beyond
# the row too.  A warm bubble and a wind lie on the end of the rows, and the halo columns hold nothing that would pass.
@pytest.mark.parametrize("nx,nz", [(3721, 8), (3721, 12), (3845, 9)])
def test_miniweather_last_segment_of_one_cell(gpx, nx, nz):
    from oracle import miniweather as mw

    segments = -(-nx // 124)
    width = -(-(-(-nx // segments)) // 4) * 4  # in whole lanes of four cells
    segments = -(-nx // width)
    assert nx - (segments - 1) * width == 1
    mw.build()
    orc = mw.Oracle(nx, nz)
    ex, be = gpx.BaseExecutor(), gpx.BLPExecutor()
    for e in (ex, be):
        e.init(f"miniweather_{nx}x{nz}")
    # (a tile of the horizontal kernel is four segments: this is the plan the widths above are of)
    assert be.model.get_kernel_info(0)["total_tiles"] == -(-nz * segments // 4)
    off = (np.arange(nx) + 0.5) / nx
    off = np.minimum(off, 1 - off)  # distance from the end of the row, around it
    bump = np.exp(-(off * nx / 6) ** 2).astype(np.float32)
    start = orc.state.copy()
    start[0, 2:-2, 2:-2] += np.float32(1e-3) * bump
    start[1, 2:-2, 2:-2] += np.float32(5.0) * bump
    start[3, 2:-2, 2:-2] += np.float32(3.0) * bump
    start[:, :, :2] = start[:, :, -2:] = -1.0
    orc.state[:] = start
    ex.model.set("state", start)
    for step in (1, 2):
        ex.execute()
        orc.timestep()
        got, want = ex.model.get("state"), orc.state
        for v, bound in enumerate((2e-6, 6e-4, 6e-4, 2e-4)):  # (as above)
            assert np.max(np.abs(mw.interior(got)[v].astype(np.float64) - mw.interior(want)[v])) <= bound * step, (step, v)
    # the same bits behind stops anywhere in the two steps
    word, s = gpx.PreemptWord(1), gpx.Stream(1)
    be.set_word(word)
    rng, stops = np.random.default_rng(nx + nz), 0
    for trial in range(6):
        be.model.set("state", start)
        for _ in range(2):
            if trial % 2:
                word.raise_()  # (launched while it is up: the first kernel is the stop)
            be.execute(s)
            for turn in range(40):
                if turn < 4:
                    until = time.perf_counter() + float(rng.uniform(0, 60e-6))
                    while time.perf_counter() < until:
                        pass
                    word.raise_()
                s.sync()
                word.clear()
                time.sleep(0.0005)
                if be.resume(s) == -1:
                    break
                stops += 1
            else:
                raise AssertionError("does not end")
            s.sync()
        assert np.array_equal(mw.interior(be.model.get("state")), mw.interior(got))
    assert stops > 0
    ex.clear(), be.clear(), word.destroy(), s.destroy()


def _same_bits_behind_stops(gpx, ex, data, names, transport, trials=8):
    """Runs of a preemptible executor that are stopped up to four times each, anywhere, end with the bits of an
    uninterrupted one."""
    word, s = gpx.PreemptWord(transport), gpx.Stream(1)
    ex.set_word(word)
    ex.set_input("data", data)
    ex.execute(s)
    s.sync()
    want = {k: ex.model.get(k) for k in names}
    t0 = time.perf_counter()
    ex.execute(s)
    s.sync()
    run = time.perf_counter() - t0
    rng, stops = np.random.default_rng(11), 0
    for _ in range(trials):
        ex.set_input("data", data * 0)
        ex.execute(s)
        s.sync()  # nothing stale can pass
        ex.set_input("data", data)
        word.clear()
        time.sleep(0.001)
        ex.execute(s)
        for turn in range(40):
            if turn < 4:
                until = time.perf_counter() + float(rng.uniform(0, run / 4))
                while time.perf_counter() < until:
                    pass
                word.raise_()
            s.sync()
            word.clear()
            time.sleep(0.0005)
            if ex.resume(s) == -1:
                break
            stops += 1
        else:
            raise AssertionError("does not end")
        s.sync()
        assert ex.error() == (0, 0)
        for k in names:
            assert np.array_equal(ex.model.get(k), want[k]), k
    assert stops > 0
    ex.clear(), word.destroy(), s.destroy()


# More rows than 32 an SM and several tiles a CTA: two tiles are claimed ahead of the one that is worked on.
@pytest.mark.parametrize("width,dtype", [(768, "float16"), (768, "float32"), (1024, "bfloat16"), (136, "float32")])
@pytest.mark.parametrize("transport", [0, 1])
def test_layernorm_of_many_rows_ends_with_the_same_bits_after_a_stop(gpx, tmp_path, width, dtype, transport):
    batch, seq = 6001, 8
    g = _Graph(batch, dtype)
    ids = g.input(batch, seq, ids=True)
    tables = [g.add(_param(k, 1.0, "table"), s) for k, s in (("word", [50, width]), ("pos", [64, width]))]
    names = ["emb"] + [f"ln{i}" for i in range(10)]
    x = None
    for name in names:
        w, b = (g.add(_param(f"{name}.{k}"), [width]) for k in ("weight", "bias"))
        x = g.op(name, "gpx_layer_norm", ([ids, *tables] if x is None else [x]) + [w, b], [batch, seq, width])
    w, b = (g.add(_param("heads." + k), [width]) for k in ("weight", "bias"))
    g.op("heads", "gpx_layer_norm", [x, w, b], [batch, seq, width])
    ex = g.load(gpx, tmp_path / "ln", gpx.BLPExecutor)
    info = ex.model.get_kernel_info(0)
    assert info["total_tiles"] > 3 * info["launch_params"][0]
    rng = np.random.default_rng(width)
    for name in names + ["heads"]:
        ex.model.set(name + ".weight", rng.normal(1, 0.1, width).astype(np.float32))
        ex.model.set(name + ".bias", rng.normal(0, 0.1, width).astype(np.float32))
    _same_bits_behind_stops(gpx, ex, rng.integers(0, 50, (batch, seq)).astype(np.int64), ["emb", "ln4", "ln9"], transport, trials=6)


# The forms beside the strips: nine taps in flight up to two tiles of 256 vectors an SM, three beyond (over rows stored
# with a border, as a 3x3 layer beside it wants them, strides from three on, up to four tiles an SM), a tap at a time.
@pytest.mark.parametrize("channels,n,hw", [(40, 1, 13), (64, 24, 56), (72, 21, 33)])
@pytest.mark.parametrize("kernel,stride,border", [(3, 1, True), (3, 2, True), (3, 3, False), (3, 2, False), (5, 1, False), (5, 2, True), (7, 1, False)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_depthwise_forms(gpx, tmp_path, channels, n, hw, kernel, stride, border, dtype):
    g = _Graph(n, dtype)
    x = g.conv("a", g.input(n, 3, hw, hw), 64 if border else channels)
    channels = g.shapes[x][1]
    if border:
        g.conv("beside", x, 64, 3, 1)
    pad = kernel // 2
    out = (hw + 2 * pad - kernel) // stride + 1
    x = g.op("b", "gpx_depthwise_conv2d", [x, g.add(_param("b.weight", 0.2), [channels, 1, kernel, kernel]), g.add(_param("b.bias"), [channels])],
             [n, channels, out, out], kernel=kernel, stride=stride, padding=pad, activation=1)
    g.heads(x)
    results = []
    for cls in (gpx.BaseExecutor, gpx.BLPExecutor):
        ex = g.load(gpx, tmp_path / cls.__name__, cls)
        s, word = gpx.Stream(1), gpx.PreemptWord(1)
        if cls is gpx.BLPExecutor:
            ex.set_word(word)
        ex.set_input("data", gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw))
        ex.execute(s)
        s.sync()
        assert ex.error() == (0, 0)
        _close(ex.model.get("b"), _conv64(ex, "b", "a", dtype, pad=pad, stride=stride, groups=channels, act=1), dtype, "b")
        results.append(ex.model.get("b"))
        ex.clear(), s.destroy(), word.destroy()
    assert np.array_equal(*results)


# Breadth-first search with as many tiles of 64 vertices as four CTAs an SM take, one more, and a last one of one vertex.
@pytest.mark.parametrize("tiles,over", [(592, 0), (592, 1), (593, 0), (700, 1)])
def test_search_tiles_around_the_resident_ctas(gpx, tmp_path, tiles, over):
    from gpreempt_b200 import graph_files
    from oracle import graphs

    graphs.build()
    prefix = str(tmp_path / "g.bel")
    graph_files.write_synthetic(prefix, tiles * 64 + over, 12, 900, 3)
    offsets, neighbours, _ = graph_files.read_bel(prefix)
    want = graphs.bfs(offsets, neighbours)[0]
    for cls in (gpx.BaseExecutor, gpx.BLPExecutor):
        ex, word, s = cls(), gpx.PreemptWord(1), gpx.Stream(1)
        ex.set_graph_path(prefix)
        ex.init("bfs")
        if cls is gpx.BLPExecutor:
            ex.set_word(word)
        ex.execute(s)
        s.sync()
        assert np.array_equal(ex.model.get("label").astype(np.uint64), np.asarray(want).astype(np.uint64))
        ex.clear(), word.destroy(), s.destroy()


# A traced latency-critical run counts the tiles of every kernel that is launched (a finishing kernel whose layer is reduced
# inside its clusters is not).
@pytest.mark.parametrize("model,dtype", [("resnet_tiny", "float32"), ("resnet50", "bfloat16"), ("mobilenet_v2", "bfloat16"), ("bert_tiny", "float16"),
                                         ("densenet_tiny", "bfloat16")])
def test_traced_latency_critical_runs_count_their_tiles(gpx, model, dtype):
    ex = gpx.BaseExecutor()
    ex.init(model, batch=1, seed=1, dtype=dtype, seq_len=16 if "bert" in model else 0)
    ex.enable_trace(True)
    ex.execute()
    gpx.device_sync()
    trace = ex.read_trace()
    for i in range(ex.get_kernel_num()):
        info = ex.model.get_kernel_info(i)
        if not (info["name"].endswith(".finish") and trace[i, 3] == 0):
            assert trace[i, 3] == info["total_tiles"], info["name"]
    ex.clear()


# Stops inside the layers behind a batch norm whose mapped operand goes to tensor memory: few K blocks, whose tiles two groups
# of epilogue warps drain in turn, and many; and float32, mapped in shared memory.
@pytest.mark.parametrize("cin", [192, 704])
@pytest.mark.parametrize("dtype,transport", [("bfloat16", 0), ("float16", 1), ("float32", 1)])
def test_batch_norm_in_the_operand_ends_with_the_same_bits_after_a_stop(gpx, tmp_path, cin, dtype, transport):
    n, hw, layers = 96, 28, 6
    g = _Graph(n, dtype, pad_channels=True)
    x = g.conv("in", g.input(n, 3, hw, hw), cin)
    for i in range(layers):
        x = g.op(f"norm{i}", "gpx_affine", [x, g.add(_param(f"norm{i}.weight"), [cin]), g.add(_param(f"norm{i}.bias"), [cin])], g.shapes[x],
                 kernel=1, stride=1, padding=0, activation=1, in_channels=cin)
        x = g.conv(f"b{i}", x, 128, act=1, std=0.06)
        if i + 1 < layers:
            x = g.conv(f"w{i}", x, cin)
    g.heads(x)
    ex = g.load(gpx, tmp_path / "norm", gpx.BLPExecutor)
    rng = np.random.default_rng(cin)
    for i in range(layers):
        ex.model.set(f"norm{i}.weight", rng.normal(1, 0.3, cin).astype(np.float32))
        ex.model.set(f"norm{i}.bias", rng.normal(0, 0.3, cin).astype(np.float32))
    _same_bits_behind_stops(gpx, ex, gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw), [f"b{i}" for i in range(layers)], transport)


@pytest.mark.parametrize("cout,cin", [(32, 128), (64, 64)])
def test_narrow_3x3_layers_in_bf16_end_with_the_same_bits_after_a_stop(gpx, tmp_path, cout, cin):
    n, hw = 24, 56
    g = _Graph(n, "bfloat16")
    x = g.conv("in", g.input(n, 3, hw, hw), cin)
    for i in range(8):
        x = g.conv(f"n{i}", x, cout, 3, 1, act=1, std=0.05)
        if cout != cin:
            x = g.conv(f"w{i}", x, cin)
    g.heads(x)
    ex = g.load(gpx, tmp_path / "be", gpx.BLPExecutor)
    _same_bits_behind_stops(gpx, ex, gpx.synth_normal(n * 3 * hw * hw, 2, 0).reshape(n, 3, hw, hw), [f"n{i}" for i in range(8)], 1)


# Two heads of eight tiles each: the last batch whose queries get a warp each on 148 SMs, and the next.
@pytest.mark.parametrize("batch", [55, 56])
def test_attention_over_few_keys_at_the_line(gpx, batch):
    test_attention_over_few_keys(gpx, batch, 64)
