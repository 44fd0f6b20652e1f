"""Forward passes of few wide rows over narrow panels, on both sides of the rule's lines, padded and cut widths, through the
operator and through training steps of layers with bias: against the double-precision oracle, and against the products
that keep a row together."""
import pytest
import torch

from conftest import abi_option, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx,base4,log_n,S,nblocks,B", [
    (1, 0, 11, 1, 1, 1), (1, 0, 11, 2, 2, 33), (1, 0, 11, 1, 1, 369), (1, 0, 11, 1, 1, 370), (1, 0, 12, 1, 2, 703), (1, 0, 13, 1, 1, 5),
    (0, 1, 12, 1, 2, 3), (0, 1, 12, 2, 1, 147), (0, 1, 13, 1, 1, 296), (0, 1, 14, 1, 2, 7), (0, 0, 12, 2, 1, 3)])
@pytest.mark.parametrize("inc,cut", [(True, 0), (False, 0), (True, 64)])
def test_few_wide_rows(oracle_mod, cplx, base4, log_n, S, nblocks, B, inc, cut):
    import butterfly_b200 as bb
    dev = torch.device("cuda", 0)
    torch.manual_seed(B)
    n, dt = 1 << log_n, torch.complex64 if cplx else torch.float32
    x = torch.randn(B, S, n - 3, dtype=dt, device=dev)
    if base4:
        tws = [torch.randn(S, nblocks, log_n // 2, n // 4, 4, 4, device=dev) / 2,
               torch.randn(S, nblocks, log_n % 2, n // 2, 2, 2, device=dev) / 2 ** 0.5]
        f = lambda: bb.butterfly_multiply_base4_fw(*tws, x, inc, n - cut)
    else:
        tw = torch.randn(S, nblocks, log_n, n // 2, 2, 2, dtype=dt, device=dev) / 2 ** 0.5
        f = lambda: bb.butterfly_multiply_fw(tw, x, inc, n - cut)
    wide = lambda t: t.detach().cpu().to(torch.complex128 if t.is_complex() else torch.float64)
    with abi_option("fw_spread", 0):
        together = f()
    y = f()
    assert rel_err(y, together) < 1e-6
    x64 = wide(x)
    ref = oracle_mod.base4_fw(*[wide(t) for t in tws], x64, inc, n - cut) if base4 else oracle_mod.multiply_fw(wide(tw), x64, inc, n - cut)
    assert rel_err(y, ref.to(dt)) < 1e-5
    layer = bb.Butterfly(n - 3, n, bias=True, complex=bool(cplx), increasing_stride=inc, nblocks=nblocks).to(dev)
    rows = x[:, 0].detach().requires_grad_(True)

    def step():
        y = layer(rows)
        return [y.detach()] + list(torch.autograd.grad(y, [rows] + list(layer.parameters()), torch.ones_like(y)))
    ltw = wide(layer.twiddle)
    d_tw, d_x = oracle_mod.multiply_bw(ltw, x64[:, :1].contiguous(), torch.ones(B, 1, n, dtype=ltw.dtype), inc)
    ly = oracle_mod.multiply_fw(ltw, x64[:, :1].contiguous(), inc)[:, 0] + wide(layer.bias)
    for got, want, what in zip(step(), (ly, d_x[:, 0], d_tw, torch.full((n,), B, dtype=ltw.dtype)), ("output", "d_input", "d_twiddle", "d_bias")):
        assert got.shape == want.shape and rel_err(got, want.to(dt)) < 1e-5, what
    assert bb.abi.device_error() == 0
