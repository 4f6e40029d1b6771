"""torch extension on the GPU: adjointness, the analytic Poisson gradient,
and the unrolled relaxed MLEM against FP64 central finite differences of the
oracle (small workload, K = 10, 64 random directions, step 1e-3 relative,
tolerance 1e-3 relative L2 over the directions)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mlem_b200 import api, synth, torch_ext  # noqa: E402

import oracle_bind as ob  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small(golden):
    m, sino, iters, gold, _ = golden.case("plain_small_it10")
    ctx = api.Context.from_matrix(m)
    yield m, sino, ctx
    ctx.close()


def test_projector_adjoint(small):
    m, sino, ctx = small
    g = torch.Generator(device="cpu").manual_seed(0)
    x = torch.rand(m.n_cols, generator=g).cuda()
    y = torch.rand(m.n_rows, generator=g).cuda()
    lhs = torch.dot(torch_ext.forward_project(x, ctx).double(), y.double())
    rhs = torch.dot(x.double(), torch_ext.back_project(y, ctx).double())
    assert abs(float(lhs - rhs)) <= 1e-5 * abs(float(lhs))
    # batched frames give the same per-frame results
    X = torch.rand(3, m.n_cols, generator=g).cuda()
    Y = torch_ext.forward_project(X, ctx)
    for b in range(3):
        assert torch.allclose(Y[b], torch_ext.forward_project(X[b].contiguous(), ctx), rtol=1e-6, atol=0)


def test_poisson_gradient_matches_analytic(small):
    m, sino, ctx = small
    x0 = synth.phantom(32, 32, 16, 5, 77).astype(np.float32) + 0.5
    x = torch.tensor(x0, device="cuda", requires_grad=True)
    s = torch.tensor(sino, device="cuda", dtype=torch.float32)
    f = torch_ext.forward_project(x, ctx)
    safe = torch.where(f > 0, f, torch.ones_like(f))
    loss = torch.sum(torch.where(f > 0, f - s * torch.log(safe), f))
    loss.backward()
    want = ob.poisson_grad_f64(m, sino, x0.astype(np.float64))
    assert ob.rel_l2(x.grad.cpu().numpy(), want) <= 1e-5


def _loss64(m, sino, x0, omega, x_true):
    xk = ob.mlem_relaxed_f64(m, sino, x0, omega)
    return float(np.mean((xk - x_true) ** 2))


@pytest.mark.parametrize("keep_bytes", [2 << 30, 0])
def test_unrolled_mlem_gradients_match_fp64_finite_differences(small, keep_bytes):
    """Both ways of the backward pass: the row sums and update factors kept
    by the forward pass, and (keep_bytes 0) recomputed from the images."""
    m, sino, ctx = small
    K = 10
    x_true = synth.phantom(32, 32, 16, 5, 0).astype(np.float64)
    norm = ob.column_sums(m)
    x0 = np.full(m.n_cols, ob.init_value(norm, sino), np.float64)
    omega = 1.0 + 0.05 * np.sin(np.arange(K))

    xt = torch.tensor(x0, device="cuda", dtype=torch.float32, requires_grad=True)
    wt = torch.tensor(omega, device="cuda", dtype=torch.float32, requires_grad=True)
    st = torch.tensor(sino, device="cuda")
    xK = torch_ext.unrolled_mlem(xt, wt, st, ctx, keep_bytes=keep_bytes)
    loss = torch.mean((xK.double() - torch.tensor(x_true, device="cuda")) ** 2)
    loss.backward()
    gx = xt.grad.double().cpu().numpy()
    gw = wt.grad.double().cpu().numpy()
    # forward agrees with the FP64 oracle
    assert ob.rel_l2(xK.detach().cpu().numpy(), ob.mlem_relaxed_f64(m, sino, x0, omega)) <= 1e-4

    rng = np.random.default_rng(1)
    eps = 1e-3
    d_gpu, d_fd = [], []
    for _ in range(64):
        v = rng.standard_normal(m.n_cols)
        v *= np.linalg.norm(x0) / np.linalg.norm(v)
        lp = _loss64(m, sino, x0 + eps * v, omega, x_true)
        lm = _loss64(m, sino, x0 - eps * v, omega, x_true)
        d_fd.append((lp - lm) / (2 * eps))
        d_gpu.append(float(gx @ v))
    d_gpu, d_fd = np.array(d_gpu), np.array(d_fd)
    assert np.linalg.norm(d_gpu - d_fd) <= 1e-3 * np.linalg.norm(d_fd)

    w_gpu, w_fd = [], []
    for _ in range(16):
        v = rng.standard_normal(K)
        v *= np.linalg.norm(omega) / np.linalg.norm(v)
        lp = _loss64(m, sino, x0, omega + eps * v, x_true)
        lm = _loss64(m, sino, x0, omega - eps * v, x_true)
        w_fd.append((lp - lm) / (2 * eps))
        w_gpu.append(float(gw @ v))
    w_gpu, w_fd = np.array(w_gpu), np.array(w_fd)
    assert np.linalg.norm(w_gpu - w_fd) <= 1e-3 * np.linalg.norm(w_fd)


@pytest.mark.parametrize("keep_bytes", [2 << 30, 0])
def test_unrolled_mlem_gradients_finite_with_tiny_projections(small, keep_bytes):
    """Rows with zero counts whose projection is tiny but nonzero (a start
    image of 1e-25: f^2 underflows to 0 in float32) give no gradient through
    calcCorrel instead of 0 / 0."""
    m, sino, ctx = small
    rng = np.random.default_rng(4)
    s = sino.copy()
    s[rng.random(s.size) < 0.3] = 0
    K = 3
    xt = torch.full((m.n_cols,), 1e-25, device="cuda", dtype=torch.float32, requires_grad=True)
    wt = torch.ones(K, device="cuda", dtype=torch.float32, requires_grad=True)
    x_true = torch.tensor(synth.phantom(32, 32, 16, 5, 0), device="cuda", dtype=torch.float32)
    xK = torch_ext.unrolled_mlem(xt, wt, torch.tensor(s, device="cuda"), ctx, keep_bytes=keep_bytes)
    loss = torch.mean((xK - x_true) ** 2)
    loss.backward()
    assert torch.isfinite(xK).all()
    assert torch.isfinite(xt.grad).all() and torch.isfinite(wt.grad).all()
    assert float(wt.grad.abs().sum()) > 0


@pytest.mark.parametrize("flags", [0, api.FLAG_NATURAL_LAYOUT | api.FLAG_NO_ROW_ORDER])
def test_backward_pass_kernels_against_the_oracle(golden, flags):
    """mlem_ratio_rows_d and mlem_adjoint_update_d (the backward pass's two
    one-pass kernels) against the oracle's projections, in the Morton layout
    with sorted rows and in natural order with file-order rows."""
    m, sino, iters, gold, _ = golden.case("plain_small_it10")
    rng = np.random.default_rng(8)
    s = np.ascontiguousarray(sino, np.int32).copy()
    s[rng.random(m.n_rows) < 0.3] = 0
    x = rng.uniform(0.5, 2.0, m.n_cols).astype(np.float32)
    du = rng.normal(0.0, 1.0, m.n_cols).astype(np.float32)
    dev = torch.device("cuda", 0)
    st = torch.cuda.current_stream().cuda_stream
    with api.Context.from_matrix(m, flags=flags) as ctx:
        xs, dus, sd = (torch.from_numpy(a).to(dev) for a in (x, du, s))
        rows = torch.empty(m.n_rows, dtype=torch.float32, device=dev)
        u = torch.empty(m.n_cols, dtype=torch.float32, device=dev)
        ctx.ratio_rows_d(xs.data_ptr(), sd.data_ptr(), rows.data_ptr(), u.data_ptr(), st)
        a = torch.empty_like(u)
        ctx.adjoint_update_d(dus.data_ptr(), sd.data_ptr(), rows.data_ptr(), a.data_ptr(), st)
        torch.cuda.synchronize()
        f_got, u_got, a_got = rows.cpu().numpy(), u.cpu().numpy(), a.cpu().numpy()
    f = ob.fwproj(m, x)
    live = s != 0
    assert ob.rel_l2(f_got[live], f[live]) <= 1e-5
    assert not f_got[~live].any()
    assert ob.rel_l2(u_got, ob.bkproj(m, ob.correl(f, s))) <= 1e-5
    f64 = f.astype(np.float64)
    dc = ob.fwproj(m, du).astype(np.float64)
    ok = live & (f64 != 0)
    df = np.where(ok, -(dc * (s / np.where(ok, f64, 1.0))) / np.where(ok, f64, 1.0), 0.0)
    assert ob.rel_l2(a_got, ob.bkproj(m, df.astype(np.float32))) <= 1e-5


def test_backward_pass_kernels_on_an_odd_matrix():
    """Empty rows, a row far longer than one load batch, duplicate columns,
    zero values and odd sizes through both backward-pass kernels."""
    from mlem_b200 import formats
    rng = np.random.default_rng(17)
    R, C = 777, 333
    lens = rng.integers(0, 40, R)
    lens[::9] = 0
    lens[5] = 10000
    row_end = np.cumsum(lens).astype(np.uint64)
    el = np.zeros(int(row_end[-1]), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, C, el.size)
    el["value"] = rng.uniform(0.0, 1.7, el.size).astype(np.float32)
    el["value"][::13] = 0.0
    m = formats.Csr4(R, C, row_end, el)
    s = rng.poisson(3.0, R).astype(np.int32)
    x = rng.uniform(0.5, 2.0, C).astype(np.float32)
    du = rng.normal(0.0, 1.0, C).astype(np.float32)
    dev = torch.device("cuda", 0)
    st = torch.cuda.current_stream().cuda_stream
    with api.Context.from_matrix(m) as ctx:
        xs, dus, sd = (torch.from_numpy(a).to(dev) for a in (x, du, s))
        rows = torch.empty(R, dtype=torch.float32, device=dev)
        u = torch.empty(C, dtype=torch.float32, device=dev)
        a = torch.empty(C, dtype=torch.float32, device=dev)
        ctx.ratio_rows_d(xs.data_ptr(), sd.data_ptr(), rows.data_ptr(), u.data_ptr(), st)
        ctx.adjoint_update_d(dus.data_ptr(), sd.data_ptr(), rows.data_ptr(), a.data_ptr(), st)
        torch.cuda.synchronize()
        f_got, u_got, a_got = rows.cpu().numpy(), u.cpu().numpy(), a.cpu().numpy()
    f = ob.fwproj(m, x)
    live = s != 0
    assert ob.rel_l2(f_got[live], f[live]) <= 1e-5
    assert ob.rel_l2(u_got, ob.bkproj(m, ob.correl(f, s))) <= 1e-5
    f64 = f.astype(np.float64)
    dc = ob.fwproj(m, du).astype(np.float64)
    ok = live & (f64 != 0)
    df = np.where(ok, -(dc * (s / np.where(ok, f64, 1.0))) / np.where(ok, f64, 1.0), 0.0)
    assert ob.rel_l2(a_got, ob.bkproj(m, df.astype(np.float32))) <= 1e-5


@pytest.mark.parametrize("n", [1, 257, 300007])
def test_relax_steps_match_tensor_expressions(n):
    """mlem_relax_step_d and mlem_relax_grad_d against the same arithmetic in
    float64: zero, negative and subnormal ratios, zero norms, one and two incoming
    gradients.  powf and logf are within 8 ulp, the products round four times:
    2^-20 relative."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    u, norm, x, g, g2 = (torch.rand(n, generator=gen, device="cuda") * 3 + 0.01 for _ in range(5))
    pick = torch.randint(0, 12, (n,), generator=gen, device="cuda")
    u[pick == 0] = 0.0
    u[pick == 1] *= -1
    norm[pick == 2] = 0.0
    u[pick == 3], norm[pick == 3] = 3e-39, 1.0
    g = g - 1.5
    el = np.zeros(1, api.ELEM_DTYPE)
    with api.Context(np.array([1], np.uint64), el, 1, n) as ctx:
        st = torch.cuda.current_stream().cuda_stream
        for w in (1.0, 0.37, 0.0):
            om = torch.tensor([w], device="cuda")
            r, xn, gx, du = (torch.empty(n, device="cuda") for _ in range(4))
            part = torch.empty(api.RELAX_PARTIALS, dtype=torch.float64, device="cuda")
            ctx.relax_step_d(x.data_ptr(), u.data_ptr(), norm.data_ptr(), om.data_ptr(), r.data_ptr(),
                             xn.data_ptr(), st)
            d = lambda t: t.double()  # noqa: E731
            rw = torch.where(norm != 0, u / torch.where(norm != 0, norm, 1.0), u)
            assert torch.equal(r, rw)
            pos = rw > 0
            want = d(x) * torch.where(pos, d(rw).clamp_min(float(np.float32(1e-38))) ** w, 0.0)
            assert torch.all((d(xn) - want).abs() <= 2.0 ** -20 * want.abs() + 1e-45)
            for second in (None, g2):
                ctx.relax_grad_d(g.data_ptr(), second.data_ptr() if second is not None else None,
                                 x.data_ptr(), r.data_ptr(), norm.data_ptr(), om.data_ptr(), gx.data_ptr(),
                                 du.data_ptr(), part.data_ptr(), st)
                gt = d(g if second is None else g + g2)
                rs = torch.where(pos, d(rw), 1.0)
                p = torch.where(pos, rs ** w, 0.0)
                dr = torch.where(pos, gt * d(x) * w * rs ** (w - 1), 0.0)
                wdu = torch.where(norm != 0, dr / torch.where(norm != 0, d(norm), 1.0), dr)
                terms = gt * d(x) * p * torch.log(rs)
                assert torch.all((d(gx) - gt * p).abs() <= 2.0 ** -20 * (gt * p).abs() + 1e-45)
                # the exponent w - 1 is rounded: log(r) 2^-24 more
                slack = 2.0 ** -20 + 2.0 ** -23 * torch.log(rs).abs()
                assert torch.all((d(du) - wdu).abs() <= slack * wdu.abs() + 1e-45)
                assert abs(float(part.sum() - terms.sum())) <= 2.0 ** -19 * float(terms.abs().sum()) + 1e-45


@pytest.mark.parametrize("where", ["g", "x"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_relax_grad_keeps_what_is_not_finite(where, value):
    """An infinite or NaN gradient or image at a voxel whose ratio is 0 shows in
    omega's gradient, as 0 times it does in the tensor expressions."""
    n = 300
    t = {k: torch.full((n,), 1.5, device="cuda") for k in ("g", "x", "r", "norm", "gx", "du")}
    om = torch.tensor([0.7], device="cuda")
    part = torch.empty(api.RELAX_PARTIALS, dtype=torch.float64, device="cuda")
    t["r"][137] = 0.0
    t[where][137] = value
    with api.Context(np.array([1], np.uint64), np.zeros(1, api.ELEM_DTYPE), 1, n) as ctx:
        ctx.relax_grad_d(t["g"].data_ptr(), None, t["x"].data_ptr(), t["r"].data_ptr(), t["norm"].data_ptr(),
                         om.data_ptr(), t["gx"].data_ptr(), t["du"].data_ptr(), part.data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
        assert part.sum().isnan()
        assert t["gx"].isnan().sum() == (where == "g") and t["du"][137] == 0.0


@pytest.mark.parametrize("keep_bytes", [2 << 30, 0])
@pytest.mark.parametrize("shape", ["K", "K1", "KC", "K1C", "norm-scalar", "norm-1C", "norm-double"])
def test_unrolled_mlem_broadcasts_omega_and_norm(shape, keep_bytes):
    """A relaxation per iteration or per voxel, and norms of other shapes and
    types: image and gradients against float64 autograd over the dense matrix.
    An iteration adds at most (40 + 60 + 10) 2^-23 relative to a positive image, and
    an image error enters the next one about threefold: 1e-4 after three; the
    gradients' terms have both signs, 1e-3 as for the finite differences above."""
    from mlem_b200 import formats
    rng = np.random.default_rng(23)
    R, C, K = 301, 157, 1 if shape in ("K1C", "norm-1C", "norm-double") else 3
    lens = rng.integers(0, 40, R)
    el = np.zeros(int(lens.sum()), formats.ELEM_DTYPE)
    el["index"] = rng.integers(0, C, el.size)
    el["value"] = rng.uniform(0.1, 1.7, el.size)
    m = formats.Csr4(R, C, np.cumsum(lens).astype(np.uint64), el)
    A = torch.zeros((R, C), dtype=torch.float64, device="cuda")
    A.index_put_((torch.from_numpy(np.repeat(np.arange(R), lens)).cuda(),
                  torch.from_numpy(el["index"].astype(np.int64)).cuda()),
                 torch.from_numpy(el["value"].astype(np.float64)).cuda(), accumulate=True)
    s = torch.from_numpy(rng.poisson(20, R).astype(np.int32)).cuda()
    om = {"KC": (K, C), "K1": (K, 1), "K1C": (K, 1, C)}.get(shape, (K,))
    omega = torch.from_numpy(rng.uniform(0.6, 1.2, om).astype(np.float32)).cuda().requires_grad_()
    x0 = torch.from_numpy(rng.uniform(0.5, 2.0, C).astype(np.float32)).cuda().requires_grad_()
    norm = {"norm-scalar": torch.tensor(17.0), "norm-1C": A.sum(0).float()[None],
            "norm-double": A.sum(0)}.get(shape, A.sum(0).float())
    with api.Context.from_matrix(m) as ctx:
        out = torch_ext.unrolled_mlem(x0, omega, s, ctx, norm=norm, keep_bytes=keep_bytes)
        v = torch.from_numpy(rng.uniform(-1.0, 2.0, tuple(out.shape)).astype(np.float32)).cuda()
        gx, gw = torch.autograd.grad((out * v.to(out.dtype)).sum(), (x0, omega))
    x64, w64, n64 = (t.detach().double().cuda() for t in (x0, omega, norm))
    x64.requires_grad_()
    w64.requires_grad_()
    x = x64
    for k in range(K):
        f = (A @ x.reshape(-1))
        c = torch.where(f != 0, s.double() / torch.where(f != 0, f, 1.0), 0.0)
        r = (A.t() @ c) / torch.where(n64 != 0, n64, 1.0)
        x = x * torch.where(r > 0, torch.where(r > 0, r, 1.0) ** w64[k], 0.0)
    hx, hw = torch.autograd.grad((x * v.double()).sum(), (x64, w64))
    assert out.shape == x.shape and gx.shape == x0.shape and gw.shape == omega.shape
    for got, want, tol in ((out, x, 1e-4), (gx, hx, 1e-3), (gw, hw, 1e-3)):
        assert float((got.detach().double() - want.detach()).norm()) <= tol * float(want.detach().norm())


@pytest.mark.parametrize("per_voxel", [False, True])
@pytest.mark.parametrize("keep_bytes", [2 << 30, 0])
def test_unrolled_mlem_under_saved_tensor_hooks(small, keep_bytes, per_voxel):
    """Hooks that hand the saved tensors back on the host, in double or strided give
    the gradients of the plain call, up to the order of float atomics."""
    m, sino, ctx = small
    s = torch.tensor(sino, device="cuda")
    hooks = [(lambda t: t, lambda t: t), (lambda t: t.cpu(), lambda t: t),
             (lambda t: t.double(), lambda t: t), (lambda t: t, lambda t: torch.stack([t, t], -1)[..., 0])]
    grads = []
    for pack, unpack in hooks:
        x0 = torch.full((m.n_cols,), 0.5, device="cuda", requires_grad=True)
        om = torch.tensor([1.0, 0.8], device="cuda")
        om = (om[:, None].repeat(1, m.n_cols) if per_voxel else om).requires_grad_()
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            x = torch_ext.unrolled_mlem(x0, om, s, ctx, keep_bytes=keep_bytes)
        grads.append(torch.autograd.grad((x * x).sum(), (x0, om)))
    for got in grads[1:]:
        for a, b in zip(got, grads[0]):
            assert float((a - b).norm()) <= 1e-5 * float(b.norm())


@pytest.mark.parametrize("frames", [2, 3, 6, 17])
def test_projections_of_several_frames_leave_no_memory_on_the_context(small, frames):
    """Their scratch is torch's: the context's device memory stays what it is, also when
    they are captured before any call has run, and the results are those of the
    interleaved entry points."""
    m = small[0]
    st = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(frames)
    with api.Context.from_matrix(m) as ctx:
        held = ctx.info.device_bytes
        for project, call, n, n_out in ((torch_ext.forward_project, ctx.fwproj_d, m.n_cols, m.n_rows),
                                        (torch_ext.back_project, ctx.bkproj_d, m.n_rows, m.n_cols)):
            v = torch.rand((frames, n), generator=gen, device="cuda")
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                captured = project(v, ctx)
            got = project(v, ctx)
            assert ctx.info.device_bytes == held
            keep = [torch.rand_like(got) for _ in range(4)]  # over the scratch that is free again
            captured.zero_()
            graph.replay()
            del graph
            vi, out = v.t().contiguous(), torch.empty((n_out, frames), device="cuda")
            call(vi.data_ptr(), out.data_ptr(), frames, st)
            assert torch.equal(got, out.t()) and torch.equal(captured, got) and len(keep) == 4
            held = ctx.info.device_bytes  # the interleaved call's own scratch stays
