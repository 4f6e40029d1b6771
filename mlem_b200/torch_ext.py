"""Differentiable MLEM for PyTorch over the same C ABI.

* `forward_project(x, ctx)`: y = A x as a torch.autograd.Function whose
  backward is the hand-written back-projection kernel (A^T g), and
  `back_project(y, ctx)` the converse.  x is float32 [C] or [B, C] on the
  context's GPU; work runs on torch's current stream.
* `unrolled_mlem(x0, omega, sino, ctx)`: K relaxed MLEM iterations
      x_{k+1} = x_k * r_k ** omega_k,  r_k = calcUpdate factor(A^T (s / A x_k), norm)
  (omega_k = 1 is the reference iteration, mlem_seq/seqcsr4mlem.cpp:163-167)
  with gradients with respect to x0 and omega.  The forward pass keeps, per
  iteration, the row sums A x_k and the update factor r_k (K x (R + C)
  floats) when they fit `keep_bytes`; the backward pass then propagates the
  adjoint through calcCorrel and both projections in one pass over the
  matrix per iteration.  Otherwise it keeps only the K images x_k
  (per-iteration checkpoints) and first recomputes A x_k and A^T(s / A x_k)
  from them in one more pass.  A context with MLEM_FLAG_MIRROR_KERNELS runs
  the same arithmetic as separate projections.

Zero rules follow the reference: the correlation is 0 where the projection
is 0 (calcCorrel), the update factor is the raw back projection where the
column sum is 0 (calcUpdate); where r_k == 0 the image entry is 0 and its
gradient with respect to omega_k is taken as 0.
"""
from __future__ import annotations

import torch

from . import api


def _check(x: torch.Tensor, n: int, what: str) -> torch.Tensor:
    if not x.is_cuda or x.dtype != torch.float32:
        raise api.MlemError(api.MLEM_ERR_INVALID, f"{what} must be a float32 CUDA tensor")
    if x.shape[-1] != n:
        raise api.MlemError(api.MLEM_ERR_INVALID, f"{what} has {x.shape[-1]} entries, expected {n}")
    return x


def _frames(x: torch.Tensor):
    """[C] -> ([C, 1], 1); [B, C] -> ([C, B] interleaved, B)."""
    if x.dim() == 1:
        return x.contiguous().view(-1, 1), 1
    return x.t().contiguous(), x.shape[0]


def _unframes(y: torch.Tensor, B: int, batched: bool):
    return y.view(-1) if not batched else y.t().contiguous()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _projected(ctx, v, n_out, frames_call, call):
    """A projection of v, [n] or [B, n], by the frame-major entry point with scratch
    from torch's allocator (an allocation of the context's own took 300 us of the first
    call on a new one, four times the call); where it finds no room, through
    interleaved copies."""
    if v.dim() == 1:
        src, out = v.contiguous(), torch.empty(n_out, dtype=torch.float32, device=v.device)
        call(src.data_ptr(), out.data_ptr(), 1, _stream())
        return out
    if v.dim() == 2 and v.shape[0] > 1:
        src = v.contiguous()
        out = torch.empty((v.shape[0], n_out), dtype=torch.float32, device=v.device)
        try:
            scratch = torch.empty(ctx.frames_scratch(v.shape[0]), dtype=torch.float32, device=v.device)
        except torch.OutOfMemoryError:
            pass
        else:
            frames_call(src.data_ptr(), out.data_ptr(), v.shape[0], _stream(), scratch.data_ptr())
            return out
    vi, B = _frames(v)
    out = torch.empty((n_out, B), dtype=torch.float32, device=v.device)
    call(vi.data_ptr(), out.data_ptr(), B, _stream())
    return _unframes(out, B, v.dim() > 1)


def _fw(ctx: "api.Context", x: torch.Tensor) -> torch.Tensor:
    return _projected(ctx, _check(x, ctx.n_cols, "image"), ctx.n_rows, ctx.fwproj_frames_d, ctx.fwproj_d)


def _bk(ctx: "api.Context", y: torch.Tensor) -> torch.Tensor:
    return _projected(ctx, _check(y, ctx.n_rows, "projection"), ctx.n_cols, ctx.bkproj_frames_d,
                      ctx.bkproj_d)


class _ForwardProject(torch.autograd.Function):
    @staticmethod
    def forward(fctx, x, ctx):
        fctx.mctx = ctx
        return _fw(ctx, x)

    @staticmethod
    def backward(fctx, g):
        return _bk(fctx.mctx, g.contiguous()), None


class _BackProject(torch.autograd.Function):
    @staticmethod
    def forward(fctx, y, ctx):
        fctx.mctx = ctx
        return _bk(ctx, y)

    @staticmethod
    def backward(fctx, g):
        return _fw(fctx.mctx, g.contiguous()), None


def forward_project(x: torch.Tensor, ctx: "api.Context") -> torch.Tensor:
    return _ForwardProject.apply(x, ctx)


def back_project(y: torch.Tensor, ctx: "api.Context") -> torch.Tensor:
    return _BackProject.apply(y, ctx)


def norm_tensor(ctx: "api.Context", device) -> torch.Tensor:
    return torch.from_numpy(ctx.column_sums()).to(device)


def _mirrored(ctx) -> bool:
    """A context with MLEM_FLAG_MIRROR_KERNELS applies the mirrors inside its
    projection kernels; the one-pass backward kernels walk full rows only."""
    return bool(ctx.info.flags & api.FLAG_MIRROR_KERNELS)


def _ratio_numerator(ctx, x, sino_i, u, f):
    """u = A^T (s / A x) and the row sums f = A x (0 for the rows without a
    count), in one pass over the matrix (mlem_ratio_rows_d).  A mirrored context
    takes the fused update and a separate forward projection instead (f is then
    A x on every row)."""
    if _mirrored(ctx):
        ctx.fused_update_d(x.data_ptr(), sino_i.data_ptr(), u.data_ptr(), 1, _stream())
        ctx.fwproj_d(x.data_ptr(), f.data_ptr(), 1, _stream())
    else:
        ctx.ratio_rows_d(x.data_ptr(), sino_i.data_ptr(), f.data_ptr(), u.data_ptr(), _stream())


def _adjoint(ctx, du, sino_i, f, out):
    """out = A^T df with df = -(A du) s / f^2 where the row has a count and f != 0:
    the adjoint of calcCorrel and both projections, in one pass
    (mlem_adjoint_update_d; a mirrored context: a forward and a back
    projection with df formed between them)."""
    if _mirrored(ctx):
        dc = _fw(ctx, du.view(-1))
        live = (sino_i != 0) & (f != 0)
        fs = torch.where(live, f, torch.ones_like(f))
        # formed as -(dc (s / f)) / f so that a tiny f never squares to 0
        df = torch.where(live, -(dc * (sino_i.to(torch.float32) / fs)) / fs, torch.zeros_like(f))
        out.copy_(_bk(ctx, df).view(out.shape))
    else:
        ctx.adjoint_update_d(du.data_ptr(), sino_i.data_ptr(), f.data_ptr(), out.data_ptr(), _stream())


def _step(ctx, x, u, norm, w, r, x_next):
    ctx.relax_step_d(x.data_ptr(), u.data_ptr(), norm.data_ptr(), w.data_ptr(), r.data_ptr(),
                     x_next.data_ptr(), _stream())


class _UnrolledMLEM(torch.autograd.Function):
    """Every iteration is one pass over the matrix and one over the voxels
    (mlem_ratio_rows_d, mlem_relax_step_d), forward and backward alike
    (mlem_relax_grad_d, mlem_adjoint_update_d)."""

    @staticmethod
    def forward(fctx, x0, omega, norm, ctx, sino_i, keep):
        K = omega.shape[0]
        x0 = x0.detach()
        xs = x0.new_empty((K,) + x0.shape)  # the images the iterations start from
        xs[0].copy_(x0)
        final, u = torch.empty_like(xs[0]), torch.empty_like(xs[0])
        kept = (torch.empty_like(xs), x0.new_empty((K, ctx.n_rows))) if keep else ()
        r, f = (None, None) if keep else (torch.empty_like(u), x0.new_empty(ctx.n_rows))
        for k in range(K):
            rk, fk = (kept[0][k], kept[1][k]) if keep else (r, f)
            _ratio_numerator(ctx, xs[k], sino_i, u, fk)
            _step(ctx, xs[k], u, norm, omega[k], rk, xs[k + 1] if k + 1 < K else final)
        fctx.mctx = ctx
        fctx.sino_i = sino_i
        fctx.keep = keep
        fctx.save_for_backward(xs, omega, norm, *kept)
        return final

    @staticmethod
    def backward(fctx, g):
        ctx = fctx.mctx
        # what saved-tensor hooks hand back, as the kernels read it
        saved = [t.to(device=g.device, dtype=torch.float32).contiguous() for t in fctx.saved_tensors]
        xs, omega, norm = saved[:3]
        K = omega.shape[0]
        g = g.contiguous()
        gx, du, out = (torch.empty_like(g) for _ in range(3))
        partial = torch.empty((K, api.RELAX_PARTIALS), dtype=torch.float64, device=g.device)
        if not fctx.keep:
            u, r, f = torch.empty_like(g), torch.empty_like(g), g.new_empty(ctx.n_rows)
        g2 = None
        for k in range(K - 1, -1, -1):
            xk = xs[k]
            if fctx.keep:  # kept by the forward pass
                r, f = saved[3][k], saved[4][k]
            else:  # recomputed from the checkpoint (du holds the unused next image)
                _ratio_numerator(ctx, xk, fctx.sino_i, u, f)
                _step(ctx, xk, u, norm, omega[k], r, du)
            # the direct path (gx) and omega's gradient, then the adjoint of A^T, of
            # calcCorrel (a row with zero counts has c = 0 whatever f is: no gradient)
            # and of A, added to the direct path by the next step
            ctx.relax_grad_d(g.data_ptr(), g2.data_ptr() if g2 is not None else None, xk.data_ptr(),
                             r.data_ptr(), norm.data_ptr(), omega[k].data_ptr(), gx.data_ptr(),
                             du.data_ptr(), partial[k].data_ptr(), _stream())
            _adjoint(ctx, du, fctx.sino_i, f, out)
            g, g2 = gx, out
        return gx + out, partial.sum(1).to(omega.dtype), None, None, None, None


class _UnrolledTensors(torch.autograd.Function):
    """The same iterations with the voxel-wise steps as tensor expressions, for
    factors and relaxations of other shapes than one float a voxel and one an
    iteration (omega[k] and norm broadcast against the image)."""

    @staticmethod
    def _ratio(ctx, x, sino_i, norm):
        x = x.to(torch.float32)  # the kernels' type, whatever the expressions' types promote to
        u, f = torch.empty_like(x), torch.empty(ctx.n_rows, dtype=torch.float32, device=x.device)
        _ratio_numerator(ctx, x, sino_i, u, f)
        return torch.where(norm != 0, u / torch.where(norm != 0, norm, torch.ones_like(norm)), u), f

    @staticmethod
    def forward(fctx, x0, omega, norm, ctx, sino_i, keep):
        xs, rs, fs = [x0.detach()], [], []
        x = x0.detach().contiguous()
        for w in omega:
            r, f = _UnrolledTensors._ratio(ctx, x, sino_i, norm)
            if keep:
                rs.append(r)
                fs.append(f)
            x = x * torch.where(r > 0, r.clamp_min(1e-38) ** w, torch.zeros_like(r))
            xs.append(x)
        fctx.mctx, fctx.sino_i, fctx.keep = ctx, sino_i, keep
        fctx.save_for_backward(torch.stack(xs[:-1]), omega, norm,
                               *([torch.stack(rs), torch.stack(fs)] if keep else []))
        return x

    @staticmethod
    def backward(fctx, g):
        ctx = fctx.mctx
        xs, omega, norm, *kept = (t.to(g.device).contiguous() for t in fctx.saved_tensors)
        g = g.contiguous()
        d_omega = torch.zeros_like(omega)
        for k in range(omega.shape[0] - 1, -1, -1):
            xk, w = xs[k].contiguous(), omega[k]
            r, f = (kept[0][k], kept[1][k]) if kept else _UnrolledTensors._ratio(ctx, xk, fctx.sino_i, norm)
            pos = r > 0
            rs = torch.where(pos, r, torch.ones_like(r))
            p = torch.where(pos, rs ** w, torch.zeros_like(r))
            term = g * (xk * p) * torch.where(pos, torch.log(rs), torch.zeros_like(r))
            d_omega[k] = term.sum_to_size(w.shape)
            dr = torch.where(pos, g * xk * w * rs ** (w - 1), torch.zeros_like(r))
            du = torch.where(norm != 0, dr / torch.where(norm != 0, norm, torch.ones_like(norm)), dr)
            du = du.to(torch.float32).contiguous()
            out = torch.empty_like(du)
            _adjoint(ctx, du, fctx.sino_i, f.to(torch.float32), out)
            g = g * p + out
        return g, d_omega, None, None, None, None


def unrolled_mlem(x0: torch.Tensor, omega: torch.Tensor, sino: torch.Tensor,
                  ctx: "api.Context", norm: torch.Tensor | None = None,
                  keep_bytes: int = 2 << 30) -> torch.Tensor:
    """K = len(omega) relaxed MLEM iterations from x0 (float32 [C] CUDA).
    omega is [K], or [K, ...] whose omega[k] broadcasts against the image: [K, C]
    holds a relaxation per voxel.  The forward pass keeps each iteration's row
    sums and update factor for the backward pass when they take at most
    keep_bytes (0: always recompute them)."""
    _check(x0, ctx.n_cols, "x0")
    if norm is None:
        norm = norm_tensor(ctx, x0.device)
    sino_i = sino.to(device=x0.device, dtype=torch.int32).contiguous()
    K = int(omega.shape[0])
    if K == 0:
        raise RuntimeError("unrolled_mlem: omega holds no iteration")
    keep = K * (ctx.n_rows + ctx.n_cols) * 4 <= keep_bytes
    omega = omega.to(device=x0.device, dtype=torch.float32)
    # The voxel-wise kernels read one relaxation an iteration and one float of x0 and
    # norm a voxel (a norm that does not broadcast to x0, or of another type or
    # device, is the tensor expressions' to take or to refuse).
    if (omega.dim() == 1 and x0.numel() == ctx.n_cols and norm.dtype == torch.float32
            and (norm.dim() == 0 or norm.device == x0.device) and norm.dim() <= x0.dim()
            and all(a in (1, b) for a, b in zip(reversed(norm.shape), reversed(x0.shape)))):
        return _UnrolledMLEM.apply(x0, omega.contiguous(), norm.to(x0.device).expand(x0.shape).contiguous(),
                                   ctx, sino_i, keep)
    return _UnrolledTensors.apply(x0, omega, norm, ctx, sino_i, keep)
