"""The bf16 GEMM where pairs of CTAs take 256 x 256 tiles: at least one 128 x 256 tile per SM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (9 * 128, 17 * 256, 64),     # odd number of row blocks: the last pair's second half is empty; one K block
    (2 * 128, 74 * 256, 192),    # one pair of row blocks, a tile for each pair of CTAs
    (13 * 128, 23 * 256, 576),   # two rounds, the second nearly empty; K blocks not a multiple of the ring
    (34 * 128, 5 * 256, 1088),   # more row blocks than one group of tiles
])
def test_pairs_match_the_oracle_and_resume_from_a_raised_word(gpx, oracle, m, n, k):
    a = oracle.f32_to_bf16(gpx.synth_uniform(m * k, 7, 0).reshape(m, k))
    b = oracle.f32_to_bf16(gpx.synth_uniform(n * k, 7, 1).reshape(n, k))
    da, db = gpx.DeviceBuffer.from_numpy(a), gpx.DeviceBuffer.from_numpy(b)
    dc = gpx.DeviceBuffer(m * n * 2)
    dc.zero()
    ctx, s, word = gpx.GemmContext(), gpx.Stream(1), gpx.PreemptWord(1)
    blp = gpx.BlpContext(word, kernel_id=3)
    word.raise_()
    gpx.gemm_bf16(da, db, dc, m, n, k, ctx, blp, s)  # the word is up: nothing runs
    s.sync()
    st = blp.read()
    assert st["stop_index"] == 3 and st["tiles_run"] == 0
    word.clear()
    blp.rearm()
    gpx.gemm_bf16(da, db, dc, m, n, k, ctx, blp, s)
    s.sync()
    st = blp.read()
    assert ctx.status() == (0, 0) and st["stop_index"] == -1 and st["tiles_run"] == gpx.gemm_tiles(m, n)
    got = oracle.bf16_to_f32(dc.download(np.uint16, m * n)).reshape(m, n).astype(np.float64)
    exact = oracle.gemm_bf16_nt(a, b)
    # half a bf16 ulp of the value plus accumulation noise
    assert np.all(np.abs(got - exact) <= np.abs(exact) * 2.0 ** -8 + np.abs(exact).max() * 1e-5)
    for o in (da, db, dc, ctx, s, word, blp):
        (o.free if hasattr(o, "free") else o.destroy)()
