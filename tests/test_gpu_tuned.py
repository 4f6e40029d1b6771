"""An autotuned context that chose the CSC method in visiting order: what that
method cannot run, or has no cut copy for, runs on the best one-pass tuning the
autotuner saw -- streamed and single host steps, and ordered subsets -- and a tuning
chosen by the caller is left alone."""
import numpy as np
import pytest

from mlem_b200 import api, synth

import oracle_bind as ob

pytestmark = pytest.mark.gpu

TOL = 1e-4


def test_autotuned_context_streams_steps_and_subsets():
    # frames enough for the two-pass method to win the autotuner's comparison
    g = synth.Geometry(64, 64, 32, 60000, 40, 200, seed=9)
    m = synth.host_matrix(g)
    rng = np.random.default_rng(2)
    sinos = [rng.poisson(4, (4, g.n_rows)).astype(np.int32) for _ in range(3)]
    for s in sinos:
        s[:, rng.random(g.n_rows) < 0.3] = 0

    def want(chain, n_after=0, subsets=1):
        out = []
        for b in range(4):
            x = None
            for s in chain:
                x = ob.mlem(m, s[b], 1, start_image=x)[0]
            if n_after:
                x = (ob.mlem(m, chain[-1][b], n_after, start_image=x)[0] if subsets == 1 else
                     ob.osem(m, chain[-1][b], n_after, subsets, start_image=x)[0])
            out.append(x)
        return out

    def close(got, ref):
        for b in range(4):
            assert ob.rel_l2(got[b], ref[b]) <= TOL

    with api.Context.from_matrix(m) as ctx:
        ctx.set_sinograms(sinos[0])
        ctx.init_images()
        chosen = ctx.autotune()
        ctx.init_images()
        ctx.iterate(2)
        close(ctx.get_images(), want([sinos[0]], 1))
        ctx.set_sinograms(sinos[0])
        ctx.init_images()
        ctx.stream_host(sinos)
        close(ctx.get_images(), want(sinos))
        ctx.iterate(2)  # no cut copy of the last sinograms
        close(ctx.get_images(), want(sinos, 2))
        x = np.ascontiguousarray(want(sinos[:1]), np.float32)
        ctx.step_host(sinos[1], x)
        close(x, want(sinos[:2]))
        ctx.set_sinograms(sinos[0])
        ctx.init_images()
        ctx.iterate(1)
        if chosen["bk_mode"] in (api.BK_CSC, api.BK_FUSED):
            ctx.set_subsets(3)
            assert ctx.kernels_per_iteration() >= 6
            ctx.iterate(2)
            close(ctx.get_images(), want(sinos[:1], 2, 3))
            ctx.set_subsets(1)
        ctx.set_tuning(api.BK_CSC, 32, 4, 8, api.VISIT_SORTED)
        ctx.set_subsets(3)
        with pytest.raises(api.MlemError):  # the caller's own choice is refused, as before
            ctx.iterate(1)


@pytest.mark.parametrize("frames", [1, 16])
@pytest.mark.parametrize("flags", [0, api.FLAG_NO_ROW_ORDER])
def test_subsets_after_autotune_whatever_it_chose(flags, frames):
    """Ordered subsets run on the one-pass tuning of an autotuned context also where the
    CSC method in file order, the atomic or the region method won the comparison."""
    g = synth.Geometry(64, 64, 32, 60000, 40, 200, seed=9)
    m = synth.host_matrix(g)
    rng = np.random.default_rng(4)
    s = rng.poisson(4, (frames, g.n_rows)).astype(np.int32)
    with api.Context.from_matrix(m, flags=flags) as ctx:
        ctx.set_sinograms(s)
        ctx.init_images()
        chosen = ctx.autotune()
        ctx.set_subsets(3)
        ctx.init_images()
        assert ctx.kernels_per_iteration() >= 6  # a pass and an update for every subset
        ctx.iterate(2)
        got = ctx.get_images()
        for b in {0, frames - 1}:
            assert ob.rel_l2(got[b], ob.osem(m, s[b], 2, 3)[0]) <= TOL
        ctx.set_subsets(1)
        assert ctx.tuning() == chosen


def test_iterations_after_streamed_steps_run_the_chosen_method():
    """mlem_iterate after streamed steps runs the method that tuning() names: the CSC
    method's sums are the same from run to run, the steps' float atomics are not."""
    g = synth.Geometry(64, 64, 32, 60000, 40, 200, seed=9)
    m = synth.host_matrix(g)
    rng = np.random.default_rng(2)
    sinos = [rng.poisson(4, (16, g.n_rows)).astype(np.int32) for _ in range(2)]
    with api.Context.from_matrix(m) as ctx:
        ctx.set_sinograms(sinos[0])
        ctx.init_images()
        start = ctx.get_images()
        if ctx.autotune()["bk_mode"] != api.BK_CSC:
            pytest.skip("the CSC method did not win the comparison here")
        got = []
        for _ in range(4):
            ctx.stream_host(sinos)
            ctx.set_images(start)
            ctx.iterate(3)
            got.append(ctx.get_images())
        assert all(np.array_equal(a, got[0]) for a in got[1:])


def captures(call):
    """Graphs instantiated by call()."""
    torch = pytest.importorskip("torch")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU,
                                            torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
    return sum(e.count for e in prof.key_averages() if e.key.startswith("cudaGraphInstantiate"))


def test_kinds_of_iterations_in_turn_keep_their_graphs():
    """Single iterations with and without statistics and host steps in turn are captured
    once each, not on every call; the streamed steps' two buffer sets, swapped after an
    odd number of them, do not leave another kind with a graph of the wrong one."""
    g = synth.Geometry(16, 16, 8, 900, 20, 60, seed=1)
    m = synth.host_matrix(g)
    rng = np.random.default_rng(6)
    s, s2 = (rng.poisson(4, (2, g.n_rows)).astype(np.int32) for _ in range(2))
    with api.Context.from_matrix(m) as ctx, api.Context.from_matrix(m) as other:
        for c in (ctx, other):
            c.set_tuning(api.BK_FUSED, 32, 1, 8, api.VISIT_SORTED)
            c.set_sinograms(s)
            c.init_images()
        x = ctx.get_images()
        batch = api.Batch([other])

        def turn():
            ctx.iterate(1, stats=True)
            ctx.iterate(1, stats=False)
            ctx.step_host(s, x)
            batch.iterate(2, stats=True)
            batch.iterate(2, stats=False)

        assert captures(lambda: (turn(), turn())) > 0
        assert captures(lambda: (turn(), turn(), turn())) == 0
        batch.close()
        for n in (1, 2, 3):  # the last sinograms in either set
            ctx.iterate(2, stats=False)
            ctx.stream_host([s2] * (n - 1) + [s])
            for stats in (True, False):
                ctx.init_images()
                ctx.iterate(2, stats=stats)
                got = ctx.get_images()
                for b in range(2):
                    assert ob.rel_l2(got[b], ob.mlem(m, s[b], 2)[0]) <= TOL


def kernels(call):
    """Names of the kernels launched by call()."""
    torch = pytest.importorskip("torch")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
    return " ".join(e.key for e in prof.key_averages())


def rows_of(lens, seed, n_cols=5000):
    from mlem_b200 import formats
    rng = np.random.default_rng(seed)
    el = np.zeros(int(lens.sum()), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, n_cols, el.size)
    el["value"] = rng.uniform(0.05, 1.7, el.size)
    return formats.Csr4(lens.size, n_cols, np.cumsum(lens).astype(np.uint64), el)


@pytest.mark.parametrize("visit", [api.VISIT_SORTED, api.VISIT_SORTED_CHUNKED])
@pytest.mark.parametrize("longest,mean,pipelined", [(256, 200, True), (400, 100, True), (401, 100, False),
                                                    (400, 200, False), (2000, 100, False)])
def test_pipelined_one_pass_walk_by_row_lengths(longest, mean, pipelined, visit):
    """The pipelined one-frame walk takes matrices whose rows fit its batch, or mostly
    do and end within five loads of it; longer rows go to the general walk.  Either
    agrees with the oracle, rows that end at and beyond the batch among them."""
    rng = np.random.default_rng(longest)
    lens = rng.integers(2 * mean - 256, 257, 6000) if mean > 128 else rng.integers(0, 2 * mean - 20, 6000)
    lens[:: 6000 // 20] = longest
    if longest > 256:
        lens[1:400:40] = 257, 287, 288, 289, 320, 352, 353, 383, 384, 399
    assert lens.max() == longest and (lens.mean() > 128) == (mean > 128)
    m = rows_of(lens, longest)
    s = rng.poisson(5, m.n_rows).astype(np.int32)
    with api.Context.from_matrix(m) as ctx:
        ctx.set_tuning(api.BK_FUSED, 32, 1, 4, visit)
        ctx.set_sinograms(s)
        ctx.init_images()
        ran = kernels(lambda: ctx.iterate(3))
        assert ("k_fused_row_one" in ran or "k_fused_chunked_one" in ran) == pipelined, ran
        assert ob.rel_l2(ctx.get_images()[0], ob.mlem(m, s, 3)[0]) <= TOL


@pytest.mark.parametrize("subsets", [1, 8])
@pytest.mark.parametrize("mean", [40, 200])
def test_depth_of_the_four_frame_walk_by_row_lengths(mean, subsets):
    """Eight elements a lane at four frames for rows longer than four hold, of the whole
    matrix or of its subsets alike."""
    rng = np.random.default_rng(mean)
    m = rows_of(rng.integers(mean - 20, mean + 21, 4000), mean)
    s = rng.poisson(5, (4, m.n_rows)).astype(np.int32)
    with api.Context.from_matrix(m) as ctx:
        ctx.set_sinograms(s)
        ctx.set_tuning(api.BK_FUSED, 32, 4, 4, api.VISIT_SORTED_CHUNKED)
        ctx.set_subsets(subsets)
        ctx.init_images()
        ran = kernels(lambda: ctx.iterate(2))
        assert ("k_fused_chunked<4, 8>" in ran) == (mean > 128), ran
        got = ctx.get_images()
    for b in (0, 3):
        ref = ob.mlem(m, s[b], 2)[0] if subsets == 1 else ob.osem(m, s[b], 2, subsets)[0]
        assert ob.rel_l2(got[b], ref) <= TOL


@pytest.mark.parametrize("rows,mean,lanes", [(300, 5, {4: 4, 8: 8, 16: 16, 32: 32}),
                                             (150000, 5, {4: 4, 8: 4, 16: 4, 32: 4}),
                                             (12000, 5, {4: 4, 8: 8, 16: 8, 32: 8}),
                                             (150000, 16, {4: 4, 8: 4, 16: 4, 32: 4}),
                                             (150000, 70, {4: 4, 8: 8, 16: 8, 32: 8})])
def test_lanes_of_the_gather_passes(rows, mean, lanes):
    """A group is the most lanes a row gets: eight where rows are many, four where they
    are also short."""
    rng = np.random.default_rng(rows)
    m = rows_of(rng.integers(1, 2 * mean, rows), rows, n_cols=rows)
    s = rng.poisson(5, rows).astype(np.int32)
    ref = ob.mlem(m, s, 2)[0]
    with api.Context.from_matrix(m) as ctx:
        for group, used in lanes.items():
            ctx.set_tuning(api.BK_CSC, group, 1, 8)
            ctx.set_sinograms(s)
            ctx.init_images()
            ran = kernels(lambda: ctx.iterate(2))
            assert f"k_fwproj<{used}, 1" in ran, (group, ran)
            assert ob.rel_l2(ctx.get_images()[0], ref) <= TOL


@pytest.mark.parametrize("rows,frames,on_device", [(601, 3, False), (25000, 1, False), (5000, 5, False),
                                                   (25001, 1, True), (5001, 5, True)])
def test_count_sums_where_they_are_cheap(rows, frames, on_device):
    """Few counts are added on the host, many on the device, to the same start value."""
    rng = np.random.default_rng(rows)
    m = rows_of(np.ones(rows, np.int64), rows, n_cols=50)
    s = rng.integers(-5, 1 << 30, (frames, rows)).astype(np.int32)
    with api.Context.from_matrix(m) as ctx:
        ran = kernels(lambda: ctx.set_sinograms(s))
        assert ("k_count_sums" in ran) == on_device, ran
        total = ctx.column_sums().astype(np.float64).cumsum()[-1]
        want = [np.float32(float(s[b].sum(dtype=np.int64)) / total) for b in range(frames)]
        assert np.array_equal(ctx.init_images(), want)


def test_start_images_need_the_sums_of_the_frames():
    """mlem_init_images after a host step with more frames than mlem_set_sinograms
    has summed is refused, not read past the sums."""
    m = rows_of(np.full(50, 3), 1, n_cols=40)
    s = np.ones((6, 50), np.int32)
    with api.Context.from_matrix(m) as ctx:
        for before in (None, s[:2]):
            if before is not None:
                ctx.set_sinograms(before)
            ctx.step_host(s, np.ones((6, 40), np.float32))
            with pytest.raises(api.MlemError) as e:
                ctx.init_images()
            assert e.value.status == api.MLEM_ERR_STATE
        ctx.set_sinograms(s)
        assert ctx.init_images().size == 6


def test_steps_of_an_autotuned_context_run_the_faster_method():
    """Host steps and streamed steps after mlem_autotune do not run the one-pass method
    where the chosen CSC method over every entry is clearly faster."""
    torch = pytest.importorskip("torch")
    g = synth.Geometry(128, 128, 64, 300000, 150, 250, seed=1)
    s = np.random.default_rng(1).poisson(4, (16, g.n_rows)).astype(np.int32)

    def ms(ctx):
        x = np.full((16, ctx.n_cols), 0.5, np.float32)
        ctx.step_host(s, x)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            ctx.step_host(s, x)
        at = {e.key: e.device_time_total for e in prof.key_averages()}
        return (sum(t for k, t in at.items() if "k_fused" in k),
                sum(t for k, t in at.items() if "k_fwproj" in k or "k_bkproj_csc" in k))

    with api.Context.siddon(g) as ctx:
        ctx.set_sinograms(s)
        ctx.init_images()
        ctx.set_tuning(api.BK_FUSED, 32, 16, 4, api.VISIT_SORTED_CHUNKED)
        one_pass = ms(ctx)[0]
        ctx.set_tuning(api.BK_CSC, 32, 16, 8, api.VISIT_SORTED)
        two_pass = ms(ctx)[1]
        ctx.set_sinograms(s)
        ctx.init_images()
        chosen = ctx.autotune()
        if chosen["bk_mode"] != api.BK_CSC or one_pass < 1.1 * two_pass:
            pytest.skip("the two methods are too close here")
        assert ms(ctx)[0] == 0


def test_four_lanes_a_row_by_frames():
    """Rows of 12 to 64 elements: four lanes in forward passes of up to eight frames, eight
    at 16 and in the back projection of columns as long."""
    rng = np.random.default_rng(5)
    m = rows_of(rng.integers(1, 80, 60000), 60000, n_cols=60000)
    for frames, lanes in ((1, 4), (4, 4), (8, 4), (16, 8)):
        s = rng.poisson(5, (frames, m.n_rows)).astype(np.int32)
        with api.Context.from_matrix(m) as ctx:
            ctx.set_sinograms(s)
            ctx.set_tuning(api.BK_CSC, 32, frames, 8)
            ctx.init_images()
            ran = kernels(lambda: ctx.iterate(2))
            assert f"k_fwproj<{lanes}, {frames}" in ran and f"k_bkproj_csc<8, {frames}>" in ran, ran
            got = ctx.get_images()
        for b in {0, frames - 1}:
            assert ob.rel_l2(got[b], ob.mlem(m, s[b], 2)[0]) <= TOL
