"""Differentiable scalar transforms for PyTorch.

`synth(sh, q)` and `analys(sh, v)` are torch.autograd.Functions over the
device transforms of a plan `sh` (shtns_b200.sht).  Their backward passes are
the hand-written adjoint kernels of the C ABI (cu_SH_to_spat_adjoint,
cu_spat_to_SH_adjoint): the adjoint of the synthesis is a quadrature-weight-
free analysis scaled by (2 - delta_m0) nphi, the adjoint of the analysis is a
synthesis weighted by the Gauss weight of each latitude.  Gradients of
complex coefficients follow PyTorch's convention dL/dRe + i dL/dIm, so the
real-valued transforms and their adjoints are exact transposes.

Inputs may be complex128/float64 (FP64) or complex64/float32 (FP32: computed
in FP64 by kernels that read and write the FP32 arrays).  Leading dimensions batch.
"""
import torch


# kinds of shtns_b200_transform: FP64, and FP32 arrays
_KIND = {"synth": (0, 8), "analys": (3, 9), "synth_adjoint": (6, 10), "analys_adjoint": (7, 11)}


def _to_spat(sh, fn, q, out, ltr):
    """fn (synthesis or adjoint of the analysis) of coefficients q into a grid
    of type out.  FP32 arrays go to the FP32 entry points as they are; any
    other pair of types is converted to FP64 and back."""
    single = q.dtype == torch.complex64 and out == torch.float32
    q = (q if single else q.to(torch.complex128)).contiguous().resolve_conj().resolve_neg()
    nf = q.numel() // sh.nlm
    v = torch.empty(tuple(q.shape[:-1]) + sh.spat_shape, dtype=torch.float32 if single else torch.float64, device=q.device)
    sh._transform(_KIND[fn][single], nf, [q], [v], ltr)
    return v.to(out)


def _to_spec(sh, fn, v, out, ltr):
    """fn (analysis or adjoint of the synthesis) of a grid v into coefficients
    of type out (types as in _to_spat)."""
    single = v.dtype == torch.float32 and out == torch.complex64
    v = (v if single else v.to(torch.float64)).contiguous().resolve_neg()
    nf = v.numel() // sh.nspat
    q = torch.empty(tuple(v.shape[:-2]) + (sh.nlm,), dtype=torch.complex64 if single else torch.complex128, device=v.device)
    sh._transform(_KIND[fn][single], nf, [v], [q], ltr)
    return q.to(out)


class _Synth(torch.autograd.Function):
    @staticmethod
    def forward(ctx, sh, q, ltr):
        ctx.sh, ctx.ltr, ctx.in_dtype = sh, ltr, q.dtype
        return _to_spat(sh, "synth", q, torch.float64 if q.dtype == torch.complex128 else torch.float32, ltr)

    @staticmethod
    def backward(ctx, g):
        return None, _to_spec(ctx.sh, "synth_adjoint", g, ctx.in_dtype, ctx.ltr), None


class _Analys(torch.autograd.Function):
    @staticmethod
    def forward(ctx, sh, v, ltr):
        ctx.sh, ctx.ltr, ctx.in_dtype = sh, ltr, v.dtype
        return _to_spec(sh, "analys", v, torch.complex128 if v.dtype == torch.float64 else torch.complex64, ltr)

    @staticmethod
    def backward(ctx, h):
        return None, _to_spat(ctx.sh, "analys_adjoint", h, ctx.in_dtype, ctx.ltr), None


def synth(sh, q, ltr=None):
    """Differentiable scalar synthesis: q (..., nlm) complex -> (..., *spat_shape)."""
    return _Synth.apply(sh, q, sh.lmax if ltr is None else int(ltr))


def analys(sh, v, ltr=None):
    """Differentiable scalar analysis: v (..., *spat_shape) real -> (..., nlm)."""
    return _Analys.apply(sh, v, sh.lmax if ltr is None else int(ltr))
