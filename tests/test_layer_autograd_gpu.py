"""The native layer operator and the fused pipelines as autograd sees them."""
import pytest
import torch
from torch.autograd import forward_ad

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda", 0)


def _layer(kind, in_size, out_size, dev, **kw):
    import butterfly_b200 as bb
    cls = bb.ButterflyBase4 if kind == "base4" else bb.Butterfly
    return cls(in_size, out_size, complex=kind == "c64", **kw).to(dev)


@pytest.mark.parametrize("kind", ["f32", "c64", "base4"])
@pytest.mark.parametrize("what", ["input", "bias", "twiddle"])
def test_layers_refuse_forward_mode(dev, kind, what):
    """No operator here has a forward-mode rule: a tangent is refused, also where no gradient is asked for."""
    layer = _layer(kind, 64, 64, dev).requires_grad_(False)
    x = torch.randn(5, 64, dtype=layer.bias.dtype, device=dev)
    with forward_ad.dual_level():
        if what == "input":
            x = forward_ad.make_dual(x, torch.randn_like(x))
        else:
            name = "twiddle4" if (kind, what) == ("base4", "twiddle") else what
            p = getattr(layer, name).detach()
            delattr(layer, name)
            setattr(layer, name, forward_ad.make_dual(p, torch.randn_like(p)))
        for grad_mode in (True, False):
            with torch.set_grad_enabled(grad_mode), pytest.raises(RuntimeError, match="jvp"):
                layer(x)


@pytest.mark.parametrize("what", ["input", "twiddle", "diagonal"])
def test_pipelines_refuse_forward_mode(dev, what):
    import butterfly_b200 as bb
    tw = torch.randn(1, 1, 6, 32, 2, 2, dtype=torch.complex64, device=dev)
    x = torch.randn(5, 1, 64, dtype=torch.complex64, device=dev)
    diag = torch.randn(64, dtype=torch.complex64, device=dev)
    with forward_ad.dual_level():
        dual = lambda name, t: forward_ad.make_dual(t, torch.randn_like(t)) if name == what else t
        with pytest.raises(RuntimeError, match="forward.mode|jvp"):
            bb.butterfly_multiply_glue(dual("twiddle", tw), dual("input", x), True, out_diag=dual("diagonal", diag))
        with pytest.raises(RuntimeError, match="forward.mode|jvp"):  # with a gradient asked for as well
            bb.butterfly_multiply_glue(dual("twiddle", tw), dual("input", x), True, out_diag=dual("diagonal", diag.requires_grad_(True)))
