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


@pytest.mark.parametrize("m,n,k", [
    (9 * 128, 17 * 256, 4096),   # empty half of the last pair; a second round that only some pairs have
    (2 * 128, 74 * 256, 8192),   # one tile for each pair: every stop is inside it
    (13 * 128, 23 * 256, 2048),  # three rounds
    (34 * 128, 40 * 256, 320),   # a K loop shorter than one grant: stops meet tile boundaries
])
@pytest.mark.parametrize("transport", [0, 1])
def test_pairs_stopped_inside_a_tile_end_with_the_same_bits(gpx, m, n, k, transport):
    """The word goes up at random times while the product runs: both CTAs of a pair stop after the same K block,
    spill, and the relaunched kernel goes on from there."""
    import time

    da, db = gpx.DeviceBuffer(m * k * 2), gpx.DeviceBuffer(n * k * 2)
    gpx.fill_uniform(da, m * k, True, 7, 0)
    gpx.fill_uniform(db, n * k, True, 7, 1)
    want, dc = gpx.DeviceBuffer(m * n * 2), gpx.DeviceBuffer(m * n * 2)
    ctx, s, word = gpx.GemmContext(), gpx.Stream(1), gpx.PreemptWord(transport)
    blp = gpx.BlpContext(word, kernel_id=3)
    gpx.gemm_bf16(da, db, want, m, n, k, ctx, blp, s)
    s.sync()
    ctx.reset(), blp.reset()
    start, end = gpx.Event(), gpx.Event()
    start.record(s)
    gpx.gemm_bf16(da, db, want, m, n, k, ctx, blp, s)
    end.record(s)
    s.sync()
    run_us = start.elapsed_ms(end) * 1e3
    rng = np.random.default_rng(m + k)
    stops = inside = 0
    for trial in range(60):
        dc.zero()
        ctx.reset(), blp.reset()
        for rounds in range(30):
            gpx.gemm_bf16(da, db, dc, m, n, k, ctx, blp, s)
            if rounds < 3:
                until = time.perf_counter() + rng.uniform(0, run_us) * 1e-6
                while time.perf_counter() < until:
                    pass
                word.raise_()
            s.sync()
            word.clear()
            gpx.device_sync()
            st = blp.read()
            if st["stop_index"] == -1:
                break
            stops += 1
            # {next iteration, K blocks done, grid} of every CTA: a CTA with K blocks stopped inside a tile
            inside += int(np.count_nonzero(ctx.buf.download(np.int32, 4 * 160, offset=64).reshape(-1, 4)[:, 1]))
            blp.rearm()
        assert ctx.status() == (0, 0) and st["stop_index"] == -1 and st["tiles_run"] == gpx.gemm_tiles(m, n), trial
        assert gpx.count_diff(want, dc, m * n * 2) == 0, trial
    assert stops > 0 and (inside > 0 or k < 512)
    for o in (da, db, dc, want, ctx, s, word, blp, start, end):
        (o.free if hasattr(o, "free") else o.destroy)()
