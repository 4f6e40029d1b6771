"""The work whose speed is followed from change to change.

Every case is a call sequence that a program using this package makes through
its public entry points: reconstructions of one or several sinograms on a
context (with the default, the command line's or the autotuned settings),
projections and unrolled reconstructions differentiated through torch,
ordered subsets, iterations streamed from host memory, and a batch over
matrices of uneven size.  The matrices are the package's synthetic Siddon
geometries; the sinograms are Poisson draws of the projections of ellipsoid
phantoms.

`exact` traces the same lines and computes the same results with plain torch
in float64, without the package.
"""
import math

import numpy as np
import torch

from mlem_b200 import api, synth, torch_ext

MIN_LEN = 1.0e-4
RADIUS_SCALE = 1.2
NO_MAX = 0xFFFFFFFF
DEV = "cuda"


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest configuration of the benchmark list (32x32x16 voxels,
        # 65,536 lines, about 20-80 elements each): one call of api.mlem with a
        # new sinogram on a context with its default settings.
        dict(name="mlem_small", kind="mlem", nx=32, ny=32, nz=16, rows=65536, lo=20, hi=80,
             frames=1, iters=10, tune="default", counts=1e7),
        # A toy scanner, as in tests and tutorials: every launch is tiny, so
        # launches and host work are what a call waits for.
        dict(name="mlem_tiny_odd", kind="mlem", nx=13, ny=11, nz=7, rows=601, lo=1, hi=NO_MAX,
             frames=3, iters=20, tune="default", counts=1e5),
        # Five dynamic frames on an odd grid, default settings.
        dict(name="mlem_frames_odd", kind="mlem", nx=75, ny=61, nz=37, rows=120007, lo=1,
             hi=NO_MAX, frames=5, iters=10, tune="default", counts=3e6),
        # The benchmark's headline: the full-size matrix, one sinogram, the
        # autotuned method, iterations on the device.
        dict(name="iterate_full", kind="iterate", nx=128, ny=128, nz=64, rows=4194304, lo=150,
             hi=250, frames=1, iters=20, tune="auto", counts=1e9),
        # What the command-line program does with the same matrix: the
        # reproducible method, sinogram in, image out.
        dict(name="mlem_full_cli", kind="mlem", nx=128, ny=128, nz=64, rows=4194304, lo=150,
             hi=250, frames=1, iters=30, tune="cli", counts=1e9),
        # Sixteen frames iterated together, autotuned (the batched benchmark
        # on a quarter of its lines).
        dict(name="iterate_frames16", kind="iterate", nx=128, ny=128, nz=64, rows=1048576, lo=150,
             hi=250, frames=16, iters=10, tune="auto", counts=5e7),
        # A forward projection and its gradient (a back projection) in torch,
        # as a learned reconstruction calls them: one image ...
        dict(name="project_1", kind="project", nx=128, ny=128, nz=64, rows=1048576, lo=150, hi=250,
             frames=1, tune="default", counts=0),
        # ... and a small batch of images on an odd grid.
        dict(name="project_6_odd", kind="project", nx=91, ny=70, nz=53, rows=300001, lo=1,
             hi=NO_MAX, frames=6, tune="default", counts=0),
        # One gradient step through five unrolled iterations (loss: mean
        # squared error of the final image).
        dict(name="unrolled_grad", kind="unrolled", nx=128, ny=128, nz=64, rows=1048576, lo=150,
             hi=250, frames=1, iters=5, tune="default", counts=2.5e8),
        # Ordered subsets, autotuned.
        dict(name="osem_8", kind="osem", nx=112, ny=96, nz=60, rows=500003, lo=100, hi=220,
             frames=1, iters=5, subsets=8, tune="auto", counts=1e8),
        # Iterations fed from page-locked host memory, one sinogram in and one
        # image out per iteration.
        dict(name="stream_host", kind="stream", nx=128, ny=128, nz=64, rows=2097152, lo=150,
             hi=250, frames=1, iters=8, tune="chunked", counts=5e8),
        # Three scanners of uneven size iterated as one batch, autotuned.
        dict(name="batch_uneven", kind="batch", nx=32, ny=32, nz=16, rows=65536, lo=20, hi=80,
             frames=12, nx2=80, ny2=72, nz2=40, rows2=250007, lo2=1, hi2=NO_MAX, frames2=7,
             nx3=128, ny3=128, nz3=64, rows3=786432, lo3=150, hi3=250, frames3=4, iters=5,
             tune="auto", counts=3e7),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid():
        if rng.random() < 0.3:  # a scanner's power-of-two grid
            return rng.choice([16, 32, 64, 128]), rng.choice([16, 32, 64, 128]), rng.choice([8, 16, 32, 64])
        return log_int(9, 128), log_int(9, 128), log_int(5, 64)

    kind = rng.choice(["mlem", "mlem", "iterate", "project", "project", "unrolled", "osem", "stream",
                       "batch"])
    nx, ny, nz = grid()
    rows = log_int(500, 1000000)
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, rows=rows, lo=1, hi=NO_MAX, frames=1)
    if rng.random() < 0.4:  # the longer lines through the grid only
        c["lo"] = (nx + ny + nz) // 4
    if kind in ("mlem", "iterate"):
        c["frames"] = rng.choice([1, 1, 1, 2, 3, 4, 6, 8, 12, 16])
        c["iters"] = rng.randint(3, 20)
        c["tune"] = rng.choice(["default", "cli", "auto"])
    elif kind == "project":
        c["frames"] = rng.choice([1, 1, 2, 3, 4, 6, 8])
        c["tune"] = "default"
    elif kind == "unrolled":
        c["iters"] = rng.randint(2, 6)
        c["tune"] = "default"
    elif kind == "osem":
        c["frames"] = rng.choice([1, 1, 2, 4])
        c["iters"] = rng.randint(2, 5)
        c["subsets"] = rng.choice([2, 4, 8, 10])
        c["tune"] = rng.choice(["chunked", "auto"])
    elif kind == "stream":
        c["frames"] = rng.choice([1, 1, 3])
        c["iters"] = rng.randint(3, 8)
        c["tune"] = "chunked"
    else:
        c["rows"] = log_int(500, 100000)
        c["frames"] = rng.choice([4, 8, 12])
        for k in ("2", "3"):
            c["nx" + k], c["ny" + k], c["nz" + k] = grid()
            c["rows" + k], c["lo" + k], c["hi" + k] = log_int(2000, 400000), 1, NO_MAX
            c["frames" + k] = rng.choice([1, 3, 4, 7])
        c["iters"] = rng.randint(2, 5)
        c["tune"] = "auto"
    c["counts"] = 50.0 * rows * 10 ** rng.uniform(-1, 1)
    return c


def _parts(case):
    """(nx, ny, nz, rows, lo, hi, frames) of every matrix of the case."""
    return [tuple(case[k + s] for k in ("nx", "ny", "nz", "rows", "lo", "hi", "frames"))
            for s in ("", "2", "3") if "nx" + s in case]


def work(case):
    total_b = total_f = 0.0
    for nx, ny, nz, rows, lo, hi, frames in _parts(case):
        c = nx * ny * nz
        if hi != NO_MAX:
            per_row = 0.46 * (lo + hi)
        else:  # the mean chord of a line through the grid, in voxels crossed
            per_row = max(float(lo), 0.4 * (nx + ny + nz))
        z = per_row * rows
        passes = {"project": 1, "unrolled": 2 * case.get("iters", 1)}.get(case["kind"], case.get("iters", 1))
        total_b += passes * (8.0 * z + 8.0 * rows + frames * (4.0 * rows + 8.0 * c))
        total_f += passes * 4.0 * z * frames
    return {"bytes": total_b, "flops": total_f}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _phantom(nx, ny, nz, n, gen):
    """Ellipsoids of intensity 1-10 on zero (float32, natural voxel order)."""
    ax = [torch.arange(m, dtype=torch.float64) + 0.5 for m in (nx, ny, nz)]
    img = torch.zeros((nz, ny, nx), dtype=torch.float32)
    dims = torch.tensor([nx, ny, nz], dtype=torch.float64)
    for _ in range(n):
        c = dims * (0.3 + 0.4 * torch.rand(3, generator=gen, dtype=torch.float64))
        a = dims * (0.08 + 0.22 * torch.rand(3, generator=gen, dtype=torch.float64))
        v = 1.0 + 9.0 * torch.rand(1, generator=gen, dtype=torch.float64)
        inside = (((ax[0] - c[0]) / a[0]) ** 2)[None, None, :] + \
            (((ax[1] - c[1]) / a[1]) ** 2)[None, :, None] + (((ax[2] - c[2]) / a[2]) ** 2)[:, None, None] <= 1.0
        img[inside] = float(v)
    return img.reshape(-1)


def _phantoms(part, seed, which):
    nx, ny, nz, _, _, _, frames = part
    gen = torch.Generator().manual_seed(1000003 * seed + 101 * which)
    return [_phantom(nx, ny, nz, 3 + int(torch.randint(0, 6, (1,), generator=gen)), gen) for _ in range(frames)]


def _counts(means, total, seed, which, frame):
    """int32 Poisson counts (on the host) of the float64 line means (on the GPU)."""
    gen = torch.Generator(device=DEV).manual_seed(7919 * seed + 31 * which + frame + 1)
    s = float(means.sum())
    lam = means * (total / s) if s > 0 else means
    return torch.poisson(lam.float(), generator=gen).to(torch.int32).cpu().numpy()


def _totals(case, frames):
    # frames of different count levels
    return [case["counts"] * 10 ** (-0.3 * f) for f in range(frames)]


def _geometry(part, seed, which):
    nx, ny, nz, rows, lo, hi, _ = part
    return synth.Geometry(nx, ny, nz, rows, lo, hi, seed=17 * seed + which, radius_scale=RADIUS_SCALE,
                          min_len=MIN_LEN)


def _tune(ctx, how):
    if how == "cli":
        t = ctx.tuning()
        ctx.set_tuning(api.BK_CSC, 32, t["frame_tile"], 8, api.VISIT_SORTED)
    elif how == "chunked":
        t = ctx.tuning()
        ctx.set_tuning(api.BK_FUSED, 32, t["frame_tile"], 4, api.VISIT_SORTED_CHUNKED)
    elif how == "auto":
        ctx.autotune()


def _scan(case, seed, which, part):
    """A context and the sinograms of its frames."""
    ctx = api.Context.siddon(_geometry(part, seed, which))
    sino = [_counts(torch.from_numpy(ctx.project_f64(x.numpy())).to(DEV), t, seed, which, f)
            for f, (x, t) in enumerate(zip(_phantoms(part, seed, which), _totals(case, part[6])))]
    return ctx, np.stack(sino)


def prepare(case, seed):
    kind, parts = case["kind"], _parts(case)
    s = dict(kind=kind, iters=case.get("iters", 1))
    if kind == "project":
        nx, ny, nz, rows, _, _, frames = parts[0]
        s["ctx"] = api.Context.siddon(_geometry(parts[0], seed, 0))
        x, g = _project_inputs(parts[0], seed)
        s["x"], s["g"] = x.float().to(DEV).requires_grad_(True), g.float().to(DEV)
        return s
    if kind == "batch":
        scans = [_scan(case, seed, k, p) for k, p in enumerate(parts)]
        for ctx, sino in scans:
            ctx.set_sinograms(sino)
            ctx.init_images()
        s["ctxs"] = [ctx for ctx, _ in scans]
        s["batch"] = api.Batch(s["ctxs"])
        s["batch"].autotune()
        return s
    ctx, sino = _scan(case, seed, 0, parts[0])
    s["ctx"] = ctx
    if kind == "unrolled":
        s["x0"] = torch.full((ctx.n_cols,), _unrolled_start(sino), device=DEV).requires_grad_(True)
        s["omega"] = _omega(case["iters"], seed).float().to(DEV).requires_grad_(True)
        s["target"] = _phantoms(parts[0], seed, 0)[0].to(DEV)
        s["sino"] = torch.from_numpy(sino[0]).to(DEV)
        s["norm"] = torch_ext.norm_tensor(ctx, DEV)
        return s
    if kind == "stream":
        # a sinogram of its own for every iteration (frames of other lengths)
        s["sinos"] = [torch.from_numpy(_streamed(sino, k)).pin_memory() for k in range(case["iters"])]
        s["images"] = [torch.empty((sino.shape[0], ctx.n_cols), dtype=torch.float32).pin_memory()
                       for _ in range(case["iters"])]
    s["sino"] = sino
    ctx.set_sinograms(sino)
    ctx.init_images()
    if kind == "osem":
        t = ctx.tuning()
        ctx.set_tuning(api.BK_FUSED, 32, t["frame_tile"], 4, api.VISIT_SORTED_CHUNKED)
        ctx.set_subsets(case["subsets"])
    _tune(ctx, case["tune"])
    return s


def _streamed(sino, k):
    return np.ascontiguousarray((sino * (3 + k % 4)) // 6)


def _project_inputs(part, seed):
    nx, ny, nz, rows, _, _, frames = part
    gen = torch.Generator().manual_seed(999 * seed + 5)
    x = torch.stack([p + 0.1 * torch.rand(p.shape, generator=gen) for p in _phantoms(part, seed, 0)])
    g = torch.randn((frames, rows), generator=gen)
    return (x[0], g[0]) if frames == 1 else (x, g)


def _unrolled_start(sino):
    return float(np.float32(0.01 + 0.02 * sino[0].mean()))


def _omega(k, seed):
    gen = torch.Generator().manual_seed(77 * seed + 3)
    return 0.9 + 0.2 * torch.rand(k, generator=gen)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "mlem":
        return api.mlem(s["ctx"], s["sino"], nIterations=s["iters"])[0]
    if kind in ("iterate", "osem"):
        s["ctx"].init_images()
        s["ctx"].iterate(s["iters"], stats=False)
        return s["ctx"].get_images()
    if kind == "stream":
        s["ctx"].init_images()
        s["ctx"].stream_host_ptr([x.data_ptr() for x in s["sinos"]], [x.data_ptr() for x in s["images"]])
        return s["images"]
    if kind == "batch":
        for ctx in s["ctxs"]:
            ctx.init_images()
        s["batch"].iterate(s["iters"], stats=False)
        return [ctx.get_images() for ctx in s["ctxs"]]
    if kind == "project":
        s["x"].grad = None
        y = torch_ext.forward_project(s["x"], s["ctx"])
        y.backward(s["g"])
        return {"y": y.detach(), "grad": s["x"].grad}
    s["x0"].grad = s["omega"].grad = None
    x = torch_ext.unrolled_mlem(s["x0"], s["omega"], s["sino"], s["ctx"], norm=s["norm"])
    ((x - s["target"]) ** 2).mean().backward()
    return {"x": x.detach(), "grad_x0": s["x0"].grad, "grad_omega": s["omega"].grad}


# ---------------------------------------------------------------------------
# The same results in 64 bits, by torch alone.
# ---------------------------------------------------------------------------
_M64 = (1 << 64) - 1


def _i64(v):
    v &= _M64
    return v - (1 << 64) if v >> 63 else v


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _mix(z):
    z = z + _i64(0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _uniform(key, k):
    salt = _mix(torch.tensor(_i64(0xD1B54A32D192ED03 * (k + 1)), dtype=torch.int64, device=key.device))
    return _shr(_mix(key ^ salt), 11).to(torch.float64) * (1.0 / 9007199254740992.0)


def _endpoint(part, seed, rows, attempt, end):
    nx, ny, nz = part[:3]
    key = _mix(_mix((rows << 8) | (attempt << 1) | end) ^ _i64(seed))
    u, v, q = (torch.full(rows.shape, f, dtype=torch.float64, device=rows.device) for f in (1.0, 0.0, 1.0))
    left = torch.arange(rows.numel(), device=rows.device)
    for t in range(64):
        a, b = 2.0 * _uniform(key[left], 2 * t) - 1.0, 2.0 * _uniform(key[left], 2 * t + 1) - 1.0
        aa, bb = a * a, b * b
        qq = aa + bb
        ok = (qq > 1.0e-12) & (qq <= 1.0)
        u[left[ok]], v[left[ok]], q[left[ok]] = a[ok], b[ok], qq[ok]
        left = left[~ok]
        if left.numel() == 0:
            break
    s = (RADIUS_SCALE * (0.5 * max(nx, ny))) / torch.sqrt(q)
    us, vs = u * s, v * s
    return 0.5 * nx + us, 0.5 * ny + vs, nz * _uniform(key, 200)


def _trace(part, seed, rows, attempt):
    """(keep [n, s], voxel [n, s], length [n, s]) of the lines, in line order."""
    dims = part[:3]
    p0 = _endpoint(part, seed, rows, attempt, 0)
    p1 = _endpoint(part, seed, rows, attempt, 1)
    n, dev = rows.numel(), rows.device
    amin, amax = torch.zeros(n, dtype=torch.float64, device=dev), torch.ones(n, dtype=torch.float64, device=dev)
    d = [b - a for a, b in zip(p0, p1)]
    miss = torch.zeros(n, dtype=torch.bool, device=dev)
    for i in range(3):
        lo, hi = (0.0 - p0[i]) / d[i], (float(dims[i]) - p0[i]) / d[i]
        flat = d[i] == 0
        miss |= flat & ((p0[i] < 0) | (p0[i] > dims[i]))
        lo, hi = torch.minimum(lo, hi), torch.maximum(lo, hi)
        amin = torch.where(flat, amin, torch.maximum(amin, lo))
        amax = torch.where(flat, amax, torch.minimum(amax, hi))
    miss |= ~(amin < amax)
    sq = [x * x for x in d]
    length = torch.sqrt((sq[0] + sq[1]) + sq[2])
    alphas, deltas = [], []
    start = torch.zeros(n, dtype=torch.int64, device=dev)
    stride = 1
    for i in range(3):
        step = amin * d[i]
        pos = p0[i] + step
        k = torch.where(d[i] < 0, torch.ceil(pos) - 1, torch.floor(pos)).clamp(0, dims[i] - 1)
        j = torch.arange(dims[i], dtype=torch.float64, device=dev)[None, :]
        up = (d[i] > 0)[:, None]
        plane = torch.where(up, k[:, None] + 1 + j, k[:, None] - j)
        a = (plane - p0[i][:, None]) / d[i][:, None]
        bad = (plane > dims[i]) | (plane < 0) | (d[i] == 0)[:, None]
        alphas.append(torch.where(bad, math.inf, a))
        deltas.append(torch.where(up, stride, -stride).to(torch.int32).expand(n, dims[i]))
        start += stride * k.to(torch.int64)
        stride *= dims[i]
    alphas.append(torch.full((n, 1), math.inf, dtype=torch.float64, device=dev))
    deltas.append(torch.zeros((n, 1), dtype=torch.int32, device=dev))
    al, order = torch.sort(torch.cat(alphas, 1), dim=1, stable=True)
    de = torch.gather(torch.cat(deltas, 1), 1, order)
    al = torch.minimum(al, amax[:, None])
    prev = torch.maximum(torch.cat([amin[:, None], al[:, :-1]], 1), amin[:, None])
    seg = (al - prev) * length[:, None]
    keep = (seg >= MIN_LEN) & ~miss[:, None]
    voxel = start[:, None] + torch.cumsum(de, 1, dtype=torch.int64) - de
    return keep, voxel, seg


def _matrix(part, seed, which, dev=DEV):
    """(row lengths int64 [R], columns int32 [Z], lengths float32 [Z]) of the geometry."""
    nx, ny, nz, rows, lo, hi, _ = part
    gseed = 17 * seed + which
    step = max(256, min(131072, (48 << 20) // (nx + ny + nz)))
    lens, cols, vals = [], [], []
    for r0 in range(0, rows, step):
        ids = torch.arange(r0, min(rows, r0 + step), dtype=torch.int64, device=dev)
        kept = torch.full(ids.shape, -1, dtype=torch.int64, device=dev)
        left = torch.arange(ids.numel(), device=dev)
        for a in range(64):
            cnt = _trace(part, gseed, ids[left], a)[0].sum(1)
            kept[left[cnt > 0]] = a
            left = left[~((cnt > 0) & (cnt >= lo) & (cnt <= hi))]
            if left.numel() == 0:
                break
        keep, voxel, seg = _trace(part, gseed, ids, kept.clamp_min(0))
        keep &= (kept >= 0)[:, None]
        lens.append(keep.sum(1))
        cols.append(voxel[keep].to(torch.int32))
        vals.append(seg[keep].to(torch.float32))
    return torch.cat(lens), torch.cat(cols), torch.cat(vals)


class _Exact:
    """A x and A^T y in float64 over chunks of rows."""

    def __init__(self, part, seed, which):
        self.len, self.col, self.val = _matrix(part, seed, which)
        self.C = part[0] * part[1] * part[2]
        end = torch.cumsum(self.len, 0)
        self.chunks, r, z, rows = [], 0, 0, self.len.numel()
        while r < rows:
            r1 = min(rows, r + (1 << 17))
            z1 = int(end[r1 - 1])
            self.chunks.append((r, r1, z, z1))
            r, z = r1, z1

    def fw(self, x):
        return torch.cat([torch.segment_reduce(self.val[z:z1].double() * x[self.col[z:z1]], "sum",
                                               lengths=self.len[r:r1], initial=0.0)
                          for r, r1, z, z1 in self.chunks])

    def bk(self, y):
        u = torch.zeros(self.C, dtype=torch.float64, device=y.device)
        for r, r1, z, z1 in self.chunks:
            u.index_add_(0, self.col[z:z1], self.val[z:z1].double() * torch.repeat_interleave(y[r:r1], self.len[r:r1]))
        return u


def _over(a, b):
    """a / b, 0 where b is 0."""
    return torch.where(b != 0, a / torch.where(b != 0, b, 1.0), 0.0)


def _factor(u, n):
    """calcUpdate's factor: u / n, u where n is 0."""
    return torch.where(n != 0, u / torch.where(n != 0, n, 1.0), u)


def _mlem_step(A, x, s, n):
    return x * _factor(A.bk(_over(s, A.fw(x))), n)


def _exact_sinos(A, case, part, seed, which):
    return [_counts(A.fw(x.to(DEV).double()), t, seed, which, f)
            for f, (x, t) in enumerate(zip(_phantoms(part, seed, which), _totals(case, part[6])))]


def _start(A, sino, norm):
    return torch.full((A.C,), float(sino.sum(dtype=np.float64)) / float(norm.sum()), dtype=torch.float64, device=DEV)


def exact(case, seed):
    kind, parts = case["kind"], _parts(case)
    out = []
    for which, part in enumerate(parts):
        A = _Exact(part, seed, which)
        rows = part[3]
        if kind == "project":
            x, g = _project_inputs(part, seed)
            x, g = x.to(DEV).double(), g.to(DEV).double()
            if part[6] == 1:
                return {"y": A.fw(x), "grad": A.bk(g)}
            return {"y": torch.stack([A.fw(v) for v in x]), "grad": torch.stack([A.bk(v) for v in g])}
        norm = A.bk(torch.ones(rows, dtype=torch.float64, device=DEV))
        sinos = _exact_sinos(A, case, part, seed, which)
        if kind == "unrolled":
            return _exact_unrolled(A, case, part, seed, sinos, norm)
        if kind == "stream":
            return _exact_stream(A, case, np.stack(sinos), norm)
        images = []
        for s in sinos:
            x, sd = _start(A, s, norm), torch.from_numpy(s).to(DEV).double()
            if kind == "osem":
                S = case["subsets"]
                mask = [(torch.arange(rows, device=DEV) % S == k).double() for k in range(S)]
                ns = [A.bk(m) for m in mask]
                for _ in range(case["iters"]):
                    for m, n in zip(mask, ns):
                        u = A.bk(_over(sd, A.fw(x)) * m)
                        x = x * torch.where(n != 0, u / torch.where(n != 0, n, 1.0), torch.where(norm != 0, 1.0, u))
            else:
                for _ in range(case["iters"]):
                    x = _mlem_step(A, x, sd, norm)
            images.append(x)
        out.append(torch.stack(images))
        del A
    return out if kind == "batch" else out[0]


def _exact_stream(A, case, sino, norm):
    xs = [_start(A, s, norm) for s in sino]
    images = []
    for k in range(case["iters"]):
        s = torch.from_numpy(_streamed(sino, k)).to(DEV).double()
        xs = [_mlem_step(A, x, si, norm) for x, si in zip(xs, s)]
        images.append(torch.stack(xs))
    return images


def _exact_unrolled(A, case, part, seed, sinos, norm):
    """K relaxed iterations and the gradients of the mean squared error."""
    s = torch.from_numpy(sinos[0]).to(DEV).double()
    omega = _omega(case["iters"], seed).to(DEV).double()
    target = _phantoms(part, seed, 0)[0].to(DEV).double()
    x = torch.full((A.C,), _unrolled_start(sinos), dtype=torch.float64, device=DEV)
    kept = []
    for w in omega:
        f = A.fw(x)
        r = _factor(A.bk(_over(s, f)), norm)
        kept.append((x, f, r))
        x = x * torch.where(r > 0, r.clamp_min(1e-300) ** w, 0.0)
    final = x
    g = 2.0 * (x - target) / x.numel()
    gw = torch.zeros_like(omega)
    for k in range(len(omega) - 1, -1, -1):
        x, f, r = kept[k]
        w, pos = omega[k], r > 0
        rs = torch.where(pos, r, 1.0)
        p = torch.where(pos, rs ** w, 0.0)
        gw[k] = (g * x * p * torch.log(rs)).sum()
        du = _factor(torch.where(pos, g * x * w * rs ** (w - 1), 0.0), norm)
        g = g * p + A.bk(_over(-_over(A.fw(du) * s, f), f))
    return {"x": final, "grad_x0": g, "grad_omega": gw}
