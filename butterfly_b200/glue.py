"""A Butterfly and the element-wise / gather modules around it as ONE kernel launch.

The reference builds its exact transforms as ``nn.Sequential`` chains -- ``FixedPermutation``
(torch_butterfly/permutation.py:65-75), ``Real2Complex`` / ``Complex2Real``
(torch_butterfly/complex_utils.py:100-122), ``Diagonal`` (torch_butterfly/diagonal.py:11-38) around
``Butterfly`` modules (torch_butterfly/special.py: fft, ifft, circulant, ...).  Every link of such a
chain reads and writes all rows in device memory.  Here the forward kernel does the links on the
tile it already holds in shared memory: the real rows are widened as they are loaded, the gather
runs inside the tile before the first factor, the diagonal and the second gather after the last
factor, and only real parts are stored when the chain ends in ``Complex2Real``.

``fuse(sequential)`` rewrites such a chain into ``ButterflyPipeline`` modules (sharing the
parameters of the original); ``butterfly_multiply_glue`` is the differentiable operator.  The
backward composes the existing operators (scatter, multiply backward, scatter): it is not fused.
Rows that do not fit a tile (n > 4096 float32, n > 2048 complex64) run link by link as before.
"""
from typing import Optional

import torch
from torch import nn

from .butterfly import Butterfly
from .complex_utils import Complex2Real, Real2Complex
from .diagonal import Diagonal
from .multiply import butterfly_multiply, butterfly_multiply_bw, butterfly_multiply_fw
from .permutation import FixedPermutation


_glue_fw = torch.ops.torch_butterfly.butterfly_multiply_glue_fw.default
_is_tracing, _transforms = torch._C._is_tracing, torch._C._functorch.peek_interpreter_stack


def _unfused(twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real):
    x = input.to(twiddle.dtype)
    if in_perm is not None:
        x = x[..., in_perm.long()]
    y = butterfly_multiply(twiddle, x, increasing_stride)
    if out_diag is not None:
        y = y * out_diag
    if out_perm is not None:
        y = y[..., out_perm.long()]
    return y.real if out_real else y


class _Glue(torch.autograd.Function):
    @staticmethod
    def forward(ctx, twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real):
        y = _glue_fw(twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real)
        if y is None:  # a shape the fused launch does not cover: the same links one by one (the backward below fits both)
            with torch.no_grad():
                y = _unfused(twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real).contiguous()
        ctx.save_for_backward(twiddle, input, in_perm, out_diag, out_perm)
        ctx.increasing_stride = increasing_stride
        return y

    @staticmethod
    def backward(ctx, grad):
        twiddle, input, in_perm, out_diag, out_perm = ctx.saved_tensors
        inc = ctx.increasing_stride
        g = grad.to(twiddle.dtype)
        if out_perm is not None:  # adjoint of the gather: scatter
            g = torch.empty_like(g).index_copy_(-1, out_perm.long(), g)
        x = input.to(twiddle.dtype)
        if in_perm is not None:
            x = x[..., in_perm.long()]
        d_diag = None
        if out_diag is not None:
            if ctx.needs_input_grad[4]:
                y = butterfly_multiply_fw(twiddle, x, inc)  # the product before the diagonal
                d_diag = (g * y.conj()).sum(dim=(0, 1)) if y.is_complex() else (g * y).sum(dim=(0, 1))
            g = g * out_diag.conj() if out_diag.is_complex() else g * out_diag
        d_twiddle, d_x = butterfly_multiply_bw(twiddle, x, g.contiguous(), inc)
        if in_perm is not None:
            d_x = torch.empty_like(d_x).index_copy_(-1, in_perm.long(), d_x)
        if not input.is_complex() and d_x.is_complex():
            d_x = d_x.real
        return d_twiddle, d_x, None, None, d_diag, None, None


def butterfly_multiply_glue(twiddle: torch.Tensor, input: torch.Tensor, increasing_stride: bool,
                            in_perm: Optional[torch.Tensor] = None, out_diag: Optional[torch.Tensor] = None,
                            out_perm: Optional[torch.Tensor] = None, out_real: bool = False) -> torch.Tensor:
    """real(  ( butterfly(twiddle) @ complex(input)[..., in_perm] * out_diag )[..., out_perm]  ), each
    link optional, as one launch.  input (batch, nstacks, n) with the dtype of twiddle, or float32
    for a complex twiddle (fewer columns than n are padded with zeros, unless they are gathered);
    in_perm / out_perm int32 vectors of n entries; out_diag n entries."""
    n = 1 << twiddle.shape[2]
    limit = 2048 if twiddle.is_complex() else 4096
    width = input.shape[-1]
    if in_perm is not None and width < n:  # the gather would read past the row, which a GPU answers with a lost context
        raise RuntimeError("butterfly_multiply_glue: in_perm needs rows of %d entries, got %d" % (n, width))
    # (a tracer and functorch's transforms see through the links, not through the fused operator's optional result)
    if n > limit or width > n or not input.is_cuda or _is_tracing() or _transforms() is not None:
        return _unfused(twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real)
    if not (torch.is_grad_enabled() and (input.requires_grad or twiddle.requires_grad
                                         or (out_diag is not None and out_diag.requires_grad))):
        y = _glue_fw(twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real)
        if y is not None:
            return y
    return _Glue.apply(twiddle, input, increasing_stride, in_perm, out_diag, out_perm, out_real)


def _rename_links(state_dict, prefix, links):
    """State saved from a chain link by link, under the names of its fused form (no-op for state saved from that form)."""
    fused = tuple(prefix + new for _, new in links if new.endswith("butterfly."))  # every pipeline has one, no link does
    if not fused or any(k.startswith(fused) for k in state_dict):
        return
    moved = {}
    for k in list(state_dict):
        for old, new in links:
            if k.startswith(prefix + old):
                moved[prefix + new + k[len(prefix + old):]] = state_dict.pop(k)
                break
    state_dict.update(moved)


class FusedChain(nn.Sequential):
    """What fuse() makes of a chain: loads the state of the fused and of the link-by-link form."""
    links = ()

    def _load_from_state_dict(self, state_dict, prefix, *args):
        _rename_links(state_dict, prefix, self.links)
        super()._load_from_state_dict(state_dict, prefix, *args)


class ButterflyPipeline(nn.Module):
    """[Real2Complex] [FixedPermutation] Butterfly [Diagonal] [FixedPermutation] [Complex2Real] as one
    module and one launch.  The Butterfly (single stack, no bias; an input narrower than n is zero-padded, an
    output narrower than n cut, where no gather or diagonal is on that side) and the Diagonal are the given
    modules, so their parameters stay shared with whoever else holds them."""

    def __init__(self, butterfly: Butterfly, in_perm: Optional[torch.Tensor] = None, diagonal: Optional[Diagonal] = None,
                 out_perm: Optional[torch.Tensor] = None, real_in: bool = False, real_out: bool = False):
        super().__init__()
        assert butterfly.nstacks == 1 and butterfly.bias is None
        assert butterfly.in_size == butterfly.n or in_perm is None
        assert butterfly.out_size == butterfly.n or (diagonal is None and out_perm is None)
        assert butterfly.complex or not (real_in or real_out)
        self.butterfly = butterfly
        self.diagonal = diagonal
        self.real_in, self.real_out = real_in, real_out
        self.register_buffer("in_perm", None if in_perm is None else in_perm.to(torch.int32))
        self.register_buffer("out_perm", None if out_perm is None else out_perm.to(torch.int32))

    #: names of the state a chain kept link by link -> names here (set by fuse)
    links = ()

    def _load_from_state_dict(self, state_dict, prefix, *args):
        _rename_links(state_dict, prefix, self.links)
        super()._load_from_state_dict(state_dict, prefix, *args)

    def forward(self, input):
        b = self.butterfly
        width = input.shape[-1]
        if width != b.n and b.in_size == b.n:  # (a narrower layer pads or trims its rows, whole ones take none but their own)
            raise RuntimeError("ButterflyPipeline: rows of %d entries expected, got %d" % (b.n, width))
        rows = input.unsqueeze(1) if input.dim() == 2 else input.reshape(-1, 1, width)
        if not self.real_in and b.complex and not rows.is_complex():
            rows = rows.to(b.twiddle.dtype)
        diag = None if self.diagonal is None else self.diagonal.diagonal
        y = butterfly_multiply_glue(b.twiddle, rows, b.increasing_stride, self.in_perm, diag, self.out_perm, self.real_out)
        if b.out_size < b.n:
            y = y[..., :b.out_size]
        return y.squeeze(1) if input.dim() == 2 else y.reshape(*input.shape[:-1], b.out_size)


def _fusible_butterfly(m) -> bool:
    return (type(m) is Butterfly and m.nstacks == 1 and m.bias is None and m.out_size <= m.n
            and m.twiddle.dtype in (torch.float32, torch.complex64))


def fuse(chain: nn.Sequential) -> nn.Sequential:
    """The same function as `chain` with every run of
    [Real2Complex] [FixedPermutation] Butterfly [Diagonal] [FixedPermutation] [Complex2Real]
    replaced by one ButterflyPipeline.  Links that do not fit the pattern are kept as they are, and so is a Butterfly of
    padded or cut rows with nothing to fold into it.  The result loads state saved from either form."""
    names, mods = list(chain._modules), list(chain)
    out, renames, i = [], [], 0
    while i < len(mods):
        j, real_in, in_perm = i, False, None
        if isinstance(mods[j], Real2Complex) and j + 1 < len(mods):
            real_in, j = True, j + 1
        links = []
        if isinstance(mods[j], FixedPermutation) and j + 1 < len(mods):
            links.append((names[j] + ".permutation", "in_perm"))
            in_perm, j = mods[j].permutation, j + 1
        b, at = mods[j], j
        fits = _fusible_butterfly(b) and (b.complex or not real_in) and (
            in_perm is None or (in_perm.shape[-1] == b.n and b.in_size == b.n))
        diagonal, out_perm, real_out = None, None, False
        if fits:
            links.append((names[j] + ".", "butterfly."))
            j += 1
            whole = b.out_size == b.n
            if whole and j < len(mods) and isinstance(mods[j], Diagonal) and mods[j].diagonal.shape == (b.n,) \
                    and mods[j].diagonal.dtype == b.twiddle.dtype:
                links.append((names[j] + ".", "diagonal."))
                diagonal, j = mods[j], j + 1
            if whole and j < len(mods) and isinstance(mods[j], FixedPermutation) and mods[j].permutation.shape[-1] == b.n:
                links.append((names[j] + ".permutation", "out_perm"))
                out_perm, j = mods[j].permutation, j + 1
            if j < len(mods) and isinstance(mods[j], Complex2Real) and b.complex:
                real_out, j = True, j + 1
            alone = i == at and j == at + 1
            fits = not alone or (b.in_size == b.n and whole)
        if not fits:
            renames.append((names[i] + ".", "%d." % len(out)))
            out.append(mods[i])
            i += 1
            continue
        pipe = ButterflyPipeline(b, in_perm, diagonal, out_perm, real_in, real_out)
        pipe.links = tuple(links)
        renames += [(old, "%d.%s" % (len(out), new)) for old, new in links]
        out.append(pipe)
        i = j
    fused = FusedChain(*out)
    fused.links = tuple(renames)
    return fused
