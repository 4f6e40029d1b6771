"""The gather passes (forward projection over rows, back projection over
columns) at the sizes where their batches, lane groups, lane rule and padded
frames turn over: rows and columns of 0, 1 and batch +- 1 elements, few long columns, many
short rows, one row far longer than the rest, and caller vectors on 4-, 8- and
16-byte boundaries, for every group and frame tile.  Every sum must lie within
the rounding of a float sum of its products: n 2^-23 sum |v x|."""
import numpy as np
import pytest

from mlem_b200 import api, formats

pytestmark = pytest.mark.gpu


def matrix(kind, rng):
    if kind == "edges":  # around multiples of every batch (lanes x depth), 1 to 384 elements
        lens = np.array([0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 47, 48, 49, 63, 64,
                         65, 95, 96, 97, 127, 128, 129, 191, 192, 193, 255, 256, 257, 383, 384, 385, 0, 0])
        R, C = lens.size, 97
    elif kind == "few-columns":  # long columns, fewer than the resident groups
        lens, R, C = np.full(20000, 6), 20000, 11
    elif kind == "many-rows":  # 8 lanes a row and a column
        lens, R, C = rng.integers(0, 5, 60000), 60000, 30000
    else:  # one row and one column far longer than a group's share
        lens = rng.integers(0, 5, 60000)
        lens[777] = 70000
        R, C = 60000, 30000
    end = np.cumsum(lens).astype(np.uint64)
    el = np.zeros(int(end[-1]), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, C, el.size)
    if kind == "one-long":
        el["index"][rng.random(el.size) < 0.3] = 4
    el["value"] = rng.uniform(-1.0, 1.7, el.size)
    return formats.Csr4(R, C, end, el, grid=(30, 40, 25) if kind == "many-rows" else (0, 0, 0))


def sums(m, x, transpose):
    """float64 sums, their magnitudes and their lengths."""
    rows = np.repeat(np.arange(m.n_rows), np.diff(np.concatenate([[0], m.row_end.astype(np.int64)])))
    cols, v = m.elems["index"].astype(np.int64), m.elems["value"].astype(np.float64)
    to, frm, n = (cols, rows, m.n_cols) if transpose else (rows, cols, m.n_rows)
    p = v[:, None] * x.astype(np.float64)[frm]
    out, mag = np.zeros((n, x.shape[1])), np.zeros((n, x.shape[1]))
    np.add.at(out, to, p)
    np.add.at(mag, to, np.abs(p))
    return out, mag, np.bincount(to, minlength=n)[:, None]


@pytest.mark.parametrize("kind", ["edges", "few-columns", "many-rows", "one-long"])
def test_gather_passes_against_float64(kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(11)
    m = matrix(kind, rng)
    st = torch.cuda.current_stream().cuda_stream
    with api.Context.from_matrix(m) as ctx:
        for B in (1, 2, 4, 8, 16, 3, 5, 12, 18):
            x, y = (rng.uniform(0.1, 1.0, (n, B)).astype(np.float32) for n in (m.n_cols, m.n_rows))
            want = {"fw": sums(m, x, False), "bk": sums(m, y, True)}
            for group in (4, 8, 16, 32):
                ctx.set_tuning(bk_mode=api.BK_CSC, group=group, frame_tile=1, blocks_per_sm=8)
                # the vectors `shift` floats past a 512-byte boundary: any float boundary at one
                # frame, 8 bytes at two and 16 at more
                for shift in (0, 1 if B % 2 else 2 if B % 4 else 4):
                    for way, src, n, call in (("fw", x, m.n_rows, ctx.fwproj_d), ("bk", y, m.n_cols, ctx.bkproj_d)):
                        a = torch.zeros(src.size + shift, device="cuda")
                        a[shift:] = torch.from_numpy(src.reshape(-1)).cuda()
                        o = torch.full((n * B + shift,), np.nan, device="cuda")
                        call(a[shift:].data_ptr(), o[shift:].data_ptr(), B, st)
                        got = o[shift:].cpu().numpy().reshape(n, B)
                        ref, mag, cnt = want[way]
                        assert np.all(np.abs(got - ref) <= 2.0 ** -23 * (cnt + 1) * mag), (way, B, group, shift)


def empty_tiles(s, tile):
    """Where all counts of the row's frame tile are 0, [R, B]."""
    R, B = s.shape
    return np.repeat(~s.reshape(R, B // tile, tile).any(axis=2), tile, axis=1)


def test_rows_without_counts_drop_what_is_not_finite():
    """calcCorrel of a row without counts in its frame tile is 0 also where its
    projection is NaN, for every tile and visit, with and without the list of rows with
    counts: such rows carry no NaN into the image."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(8)
    R, C = 3000, 2000
    lens = rng.integers(1, 5, R)
    el = np.zeros(int(lens.sum()), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, C, el.size)
    el["value"] = rng.uniform(0.1, 1.7, el.size)
    m = formats.Csr4(R, C, np.cumsum(lens).astype(np.uint64), el)
    A = np.zeros((R, C), bool)
    A[np.repeat(np.arange(R), lens), el["index"]] = True
    bad = rng.random(C) < 0.05
    hit = A[:, bad].any(axis=1)
    st = torch.cuda.current_stream().cuda_stream
    for flags in (0, api.FLAG_NO_ROW_ORDER):
        with api.Context.from_matrix(m, flags=flags) as ctx:
            for B in (1, 2, 4, 8, 16, 32):
                s = rng.poisson(2, (R, B)).astype(np.int32)
                s[rng.random(R) < 0.5] = 0
                s[::3, : B // 2] = 0
                x = np.where(bad[:, None], np.nan, rng.uniform(0.5, 2.0, (C, B))).astype(np.float32)
                xd, sd = torch.from_numpy(x).cuda(), torch.from_numpy(s).cuda()
                c = torch.empty((R, B), device="cuda")
                ctx.fwproj_correl_d(xd.data_ptr(), sd.data_ptr(), c.data_ptr(), B, st)
                want = hit[:, None] & ~empty_tiles(s, min(B, 16))
                assert np.array_equal(np.isnan(c.cpu().numpy()), want), B
                assert not c.cpu().numpy()[empty_tiles(s, min(B, 16))].any()
                # no tuning chosen: the widest tile, each frame on its own
                with api.Context.from_matrix(m, flags=flags) as own:
                    own.set_sinograms(np.ascontiguousarray(s.T))
                    assert own.tuning()["frame_tile"] == min(B, 16)
                    own.set_images(np.ascontiguousarray(x.T))
                    own.iterate(1)
                    ref = bad[:, None] | (A.T.astype(np.float32) @ (hit[:, None] & (s != 0)).astype(np.float32) > 0)
                    assert np.array_equal(np.isnan(own.get_images().T), ref), (B, flags)
                for tile in (t for t in (1, 2, 4, 8, 16) if t <= B):
                    for visit in (api.VISIT_FILE,) + (() if flags else (api.VISIT_SORTED,)):
                        ctx.set_sinograms(np.ascontiguousarray(s.T))
                        ctx.set_tuning(api.BK_CSC, 32, tile, 8, visit)
                        ctx.set_images(np.ascontiguousarray(x.T))
                        ctx.iterate(1)
                        nan_rows = hit[:, None] & ~empty_tiles(s, tile)
                        ref = bad[:, None] | (A.T.astype(np.float32) @ nan_rows.astype(np.float32) > 0)
                        assert np.array_equal(np.isnan(ctx.get_images().T), ref), (B, tile, visit, flags)


def test_default_frame_tile_follows_the_frames():
    """Without a chosen tuning the frame tile is the widest one of the frame
    count; a chosen one stays."""
    rng = np.random.default_rng(3)
    m = matrix("many-rows", rng)
    m.elems["value"] = np.abs(m.elems["value"])
    sino = rng.poisson(5, (5, m.n_rows)).astype(np.int32)
    imgs = []
    for tile in (None, 1):
        with api.Context.from_matrix(m) as ctx:
            ctx.set_sinograms(sino)
            assert ctx.tuning()["frame_tile"] == 8
            if tile:
                ctx.set_tuning(api.BK_CSC, 32, tile, 8)
            ctx.set_sinograms(sino[:1])
            assert ctx.tuning()["frame_tile"] == 1
            ctx.set_sinograms(sino)
            assert ctx.tuning()["frame_tile"] == (tile or 8)
            ctx.init_images()
            ctx.iterate(4)
            imgs.append(ctx.get_images().astype(np.float64))
    assert np.linalg.norm(imgs[0] - imgs[1]) <= 1e-5 * np.linalg.norm(imgs[1])


@pytest.mark.parametrize("visit", [api.VISIT_SORTED, api.VISIT_SORTED_CHUNKED])
@pytest.mark.parametrize("rows", [2, 33, 12000])
def test_pipelined_one_pass_against_float64(visit, rows):
    """The one-frame sorted one-pass walk at the edges of its 256-element batch,
    with fewer and more rows than warps: u = A^T (s / A x), each entry within the
    rounding of its terms."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(rows)
    edges = np.array([0, 1, 31, 32, 33, 255, 256, 257, 287, 288, 511, 512, 513, 900, 4096])
    lens = edges[rng.integers(0, edges.size, rows)] if rows > 100 else edges[np.arange(rows) % edges.size]
    lens[-1] = 257
    end = np.cumsum(lens).astype(np.uint64)
    C = 5000
    el = np.zeros(int(end[-1]), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, C, el.size)
    el["value"] = rng.uniform(0.05, 1.7, el.size)
    m = formats.Csr4(rows, C, end, el)
    s = rng.poisson(3, rows).astype(np.int32)
    x = rng.uniform(0.1, 2.0, C).astype(np.float32)
    f = sums(m, x[:, None], False)[0][:, 0]
    c = np.where(f != 0, s / np.where(f != 0, f, 1.0), 0.0)
    ref, mag, cnt = sums(m, c[:, None], True)
    with api.Context.from_matrix(m) as ctx:
        ctx.set_tuning(api.BK_FUSED, 32, 1, 4, visit)
        xd, sd = torch.from_numpy(x).cuda(), torch.from_numpy(s).cuda()
        for own in (False, True):  # the caller's sinogram over every row, the context's over its list
            u = torch.full((C,), np.nan, device="cuda")
            if own:
                ctx.set_sinograms(s)
            ctx.fused_update_d(xd.data_ptr(), 0 if own else sd.data_ptr(), u.data_ptr(), 1,
                               torch.cuda.current_stream().cuda_stream)
            got = u.cpu().numpy().astype(np.float64)
            # n terms, each with its factor's error: a sum of at most 4096 products and a division
            assert np.all(np.abs(got - ref[:, 0]) <= 2.0 ** -23 * (cnt[:, 0] + 4096 + 4) * mag[:, 0])


@pytest.mark.parametrize("visit", [api.VISIT_FILE, api.VISIT_SORTED, api.VISIT_SORTED_CHUNKED])
@pytest.mark.parametrize("long_rows", [False, True])
def test_four_frame_one_pass_against_float64(visit, long_rows):
    """The one-pass walks at four frames at the edges of their 4-, 6- and 8-element
    batches (128, 192 and 256 elements a row), with mean row lengths on both sides of
    128: u = A^T (s / A x), each entry within the rounding of its terms."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    R, C, B = 4000, 5000, 4
    lens = rng.choice([0, 1, 31, 33, 127, 128, 129] + [191, 192, 193, 255, 256] * (2 * long_rows), R)
    assert (lens.mean() > 128) == long_rows
    end = np.cumsum(lens).astype(np.uint64)
    el = np.zeros(int(end[-1]), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, C, el.size)
    el["value"] = rng.uniform(0.05, 1.7, el.size)
    m = formats.Csr4(R, C, end, el)
    s = rng.poisson(3, (R, B)).astype(np.int32)
    x = rng.uniform(0.1, 2.0, (C, B)).astype(np.float32)
    f = sums(m, x, False)[0]
    c = np.where(f != 0, s / np.where(f != 0, f, 1.0), 0.0)
    ref, mag, cnt = sums(m, c, True)
    with api.Context.from_matrix(m) as ctx:
        ctx.set_tuning(api.BK_FUSED, 32, 4, 4, visit)
        xd, sd = torch.from_numpy(x).cuda(), torch.from_numpy(s).cuda()
        u = torch.full((C, B), np.nan, device="cuda")
        ctx.fused_update_d(xd.data_ptr(), sd.data_ptr(), u.data_ptr(), B,
                           torch.cuda.current_stream().cuda_stream)
        got = u.cpu().numpy().astype(np.float64)
    # n terms, each with its factor's error: a sum of at most 256 products and a division
    assert np.all(np.abs(got - ref) <= 2.0 ** -23 * (cnt + 256 + 4) * mag)


@pytest.mark.parametrize("flags", [0, api.FLAG_NATURAL_LAYOUT, api.FLAG_NO_CSC])
def test_frame_major_projections(flags):
    """mlem_fwproj_frames_d / mlem_bkproj_frames_d against the interleaved entry
    points, padded and unpadded frame counts: the same kernels over the same
    device vectors, so the same bits (within rounding where rows are scattered)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    m = matrix("many-rows", rng)
    st = torch.cuda.current_stream().cuda_stream
    with api.Context.from_matrix(m, flags=flags) as ctx:
        for B in (1, 2, 3, 6, 16, 19):
            for n_in, n_out, frames, inter in ((m.n_cols, m.n_rows, ctx.fwproj_frames_d, ctx.fwproj_d),
                                               (m.n_rows, m.n_cols, ctx.bkproj_frames_d, ctx.bkproj_d)):
                v = torch.from_numpy(rng.uniform(0.1, 1.0, (B, n_in)).astype(np.float32)).cuda()
                a = torch.full((B, n_out), np.nan, device="cuda")
                b = torch.full((n_out, B), np.nan, device="cuda")
                frames(v.data_ptr(), a.data_ptr(), B, st)
                vi = v.t().contiguous()
                inter(vi.data_ptr(), b.data_ptr(), B, st)
                if flags & api.FLAG_NO_CSC and n_in == m.n_rows:
                    assert torch.allclose(a, b.t(), rtol=1e-4, atol=1e-5)
                else:
                    assert torch.equal(a, b.t())


def test_frame_scratch_on_two_streams_and_under_capture():
    """Projections of several frames on two streams take turns with the context's
    scratch, and a captured one does not use it: replayed after a call that replaces
    the scratch it still gives its own result."""
    torch = pytest.importorskip("torch")
    from mlem_b200 import torch_ext
    rng = np.random.default_rng(6)
    m = matrix("many-rows", rng)
    m = formats.Csr4(m.n_rows, m.n_cols, m.row_end, m.elems)  # no grid: no voxel scratch either
    with api.Context.from_matrix(m) as ctx:
        v = [torch.from_numpy(rng.uniform(0.1, 1.0, (3, m.n_cols)).astype(np.float32)).cuda() for _ in range(2)]
        ref = [torch_ext.forward_project(t, ctx) for t in v]
        side = [torch.cuda.Stream() for _ in v]
        torch.cuda.synchronize()
        got = [[], []]
        for _ in range(20):
            for i, s in enumerate(side):
                with torch.cuda.stream(s):
                    got[i].append(torch_ext.forward_project(v[i], ctx))
        torch.cuda.synchronize()
        assert all(torch.equal(g, ref[i]) for i in (0, 1) for g in got[i])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = torch_ext.forward_project(v[0], ctx)
        torch_ext.forward_project(torch.rand((16, m.n_cols), device="cuda"), ctx)  # a larger scratch
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        # rows of at most 4 products below 1.7: n 2^-23 sum |v x|
        assert torch.allclose(out, ref[0], rtol=0, atol=4 * 6.8 * 2.0 ** -23)


@pytest.mark.parametrize("kind", ["many-rows", "long-rows", "mirrored"])
def test_device_calls_on_two_streams_and_under_capture(kind):
    """The device-pointer calls of a context with a grid (voxel scratch), with long rows
    and with mirrored kernels (row scratch) on two streams, and two captured ones replayed
    on two streams beside eager calls that make the scratch grow: each gives what it gives
    alone, and none spoils the calls after it.  Float atomics: 1e-5 relative."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(13)
    if kind == "mirrored":
        from test_symmetry_oracle import sym_matrix
        m = sym_matrix(7, seed=3, grid=(8, 8, 4))
    else:
        m = matrix("many-rows", rng)
        if kind == "long-rows":
            lens = np.diff(np.concatenate([[0], m.row_end.astype(np.int64)]))
            lens[[5, 70]] = 40000
            el = np.zeros(int(lens.sum()), formats.ELEM_DTYPE)
            el["index"] = rng.integers(0, m.n_cols, el.size)
            el["value"] = rng.uniform(0.1, 1.7, el.size)
            m = formats.Csr4(m.n_rows, m.n_cols, np.cumsum(lens).astype(np.uint64), el, grid=(30, 40, 25))
    with (api.Context.symmetric(m, flags=api.FLAG_MIRROR_KERNELS) if kind == "mirrored" else
          api.Context.from_matrix(m)) as ctx:
        R, C = ctx.n_rows, ctx.n_cols
        gen = torch.Generator(device="cuda").manual_seed(1)

        def rand(*shape):
            return torch.rand(shape, generator=gen, device="cuda") + 0.1

        def calls(B):
            x, y, s = rand(C, B), rand(R, B), torch.randint(0, 4, (R, B), generator=gen, device="cuda", dtype=torch.int32)
            f = [(R, lambda o, st: ctx.fwproj_d(x.data_ptr(), o.data_ptr(), B, st)),
                 (C, lambda o, st: ctx.bkproj_d(y.data_ptr(), o.data_ptr(), B, st)),
                 (R, lambda o, st: ctx.fwproj_correl_d(x.data_ptr(), s.data_ptr(), o.data_ptr(), B, st)),
                 (C, lambda o, st: ctx.fused_update_d(x.data_ptr(), s.data_ptr(), o.data_ptr(), B, st))]
            if B == 1 and kind != "mirrored":
                f += [(C, lambda o, st: ctx.adjoint_update_d(x.data_ptr(), s.data_ptr(), y.data_ptr(), o.data_ptr(), st))]
            return [(torch.empty((n, B), device="cuda"), g) for n, g in f]

        def close(a, b):
            return float((a - b).norm()) <= 1e-5 * float(b.norm())

        here = torch.cuda.current_stream().cuda_stream
        sets = [calls(1), calls(1)]
        refs = []
        for one in sets:
            refs.append([])
            for o, g in one:
                g(o, here)
                refs[-1].append(o.clone())
        side = [torch.cuda.Stream() for _ in sets]
        torch.cuda.synchronize()
        for _ in range(10):
            for (k, (a, ga)), (b, gb) in zip(enumerate(sets[0]), reversed(sets[1])):
                for o, g, q in ((a, ga, side[0]), (b, gb, side[1])):
                    with torch.cuda.stream(q):
                        o.zero_()
                        g(o, q.cuda_stream)
        torch.cuda.synchronize()
        assert all(close(o, r) for one, ref in zip(sets, refs) for (o, _), r in zip(one, ref))
        graphs = []
        for one, q in zip(sets, side):
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1], stream=q):
                for o, g in one:
                    g(o, q.cuda_stream)
        for o, g in calls(5) + calls(16):  # the eager calls' scratch grows
            g(o, here)
        torch.cuda.synchronize()
        for _ in range(10):
            for one, graph, q in zip(sets, graphs, side):
                with torch.cuda.stream(q):
                    for o, _ in one:
                        o.zero_()
                    graph.replay()
            for o, g in calls(2):
                g(o, here)
        torch.cuda.synchronize()
        assert all(close(o, r) for one, ref in zip(sets, refs) for (o, _), r in zip(one, ref))
        for one, ref in zip(sets, refs):
            for (o, g), r in zip(one, ref):
                o.zero_()
                g(o, here)
                assert close(o, r)
        del graphs
