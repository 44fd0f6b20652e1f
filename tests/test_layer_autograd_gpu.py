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


@pytest.mark.parametrize("kind,in_size,out_size,lead,bias", [
    ("f32", 64, 64, (3, 5), True), ("f32", 64, 64, (7,), True), ("f32", 64, 100, (7,), True), ("f32", 64, 50, (2, 7), False), ("c64", 64, 50, (7,), True),
    ("c64", 64, 64, (3, 4), True), ("base4", 64, 50, (7,), True), ("base4", 64, 64, (), True)])
def test_layer_outputs_take_in_place_operators(dev, kind, in_size, out_size, lead, bias):
    """nn.ReLU(inplace=True) behind a layer: whatever the rank and the cut, the output is a tensor of its own."""
    torch.manual_seed(3)
    layer = _layer(kind, in_size, out_size, dev, bias=bias)
    x = torch.randn(*lead, in_size, dtype=torch.complex64 if kind == "c64" else torch.float32, device=dev, requires_grad=True)
    scale = torch.randn(*lead, out_size, dtype=x.dtype, device=dev)

    def grads(in_place):
        y = layer(x)
        assert y.shape == scale.shape and not y._is_view()
        z = y.mul_(scale) if in_place else y * scale
        return [z.detach().clone()] + list(torch.autograd.grad(z.abs().sum(), [x] + list(p for p in layer.parameters() if p.numel())))
    for a, b in zip(grads(True), grads(False)):
        assert a.shape == b.shape and (a - b).abs().max() <= 1e-5 * b.abs().max()


@pytest.mark.parametrize("kind,in_size,out_size", [("f32", 100, 70), ("f32", 40, 3000), ("c64", 60, 50), ("base4", 100, 128)])
@pytest.mark.parametrize("batch", [64, 65, 700, 2048, 2049, 40011])
def test_bias_gradients_have_one_order(dev, kind, in_size, out_size, batch):
    """The bias gradient of a layer off the fused route sums its rows in an order that the shape fixes: the same bits on
    every call, the float64 sum within what float32 sums of that many rows may be off (terms that grow like the square root of the rows, 2^-24 of the sum so far each)."""
    torch.manual_seed(batch)
    layer = _layer(kind, in_size, out_size, dev)
    x = torch.randn(batch, in_size, dtype=layer.bias.dtype, device=dev)
    g = torch.randn(batch, out_size, dtype=layer.bias.dtype, device=dev)
    first = torch.autograd.grad(layer(x), [layer.bias], g)[0]
    for _ in range(10):
        assert torch.equal(torch.autograd.grad(layer(x), [layer.bias], g)[0], first)
    wide = torch.complex128 if kind == "c64" else torch.float64
    want = g.to(wide).sum(0)
    assert (first.to(wide) - want).abs().max() <= 2e-6 * want.abs().max()


@pytest.mark.parametrize("kind", ["f32", "c64", "base4"])
def test_glue_given_to_a_class_later_runs(dev, kind, monkeypatch):
    """pre_process / post_process are looked up at the call, as methods are."""
    import butterfly_b200 as bb
    layer = _layer(kind, 60, 50, dev)
    x = torch.randn(7, 60, dtype=layer.bias.dtype, device=dev)
    plain, bias = layer(x).detach(), layer.bias.detach()
    pre, post = bb.Butterfly.pre_process, bb.Butterfly.post_process
    cls = type("Own", (type(layer),), {})
    layer.__class__ = cls
    assert torch.equal(layer(x), plain)
    cls.pre_process = lambda self, rows: pre(self, 2 * rows)
    assert torch.allclose(layer(x), 2 * (plain - bias) + bias, rtol=1e-4, atol=1e-4)
    del cls.pre_process
    cls.post_process = lambda self, rows, out, out_size=None: 3 * post(self, rows, out, out_size)
    assert torch.allclose(layer(x), 3 * plain, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("kind", ["c64", "base4"])
@pytest.mark.parametrize("bias", ["promoted", "broadcast"])
def test_biases_that_promote_or_broadcast(dev, kind, bias):
    """Complex and radix-4 layers add whatever bias PyTorch adds to their output."""
    layer = _layer(kind, 60, 50, dev)
    x = torch.randn(7, 60, dtype=layer.bias.dtype, device=dev)
    own = layer.bias.detach().clone()
    base = layer(x).detach() - own
    new = torch.randn(50, dtype=torch.float32 if kind == "c64" else torch.float64, device=dev) if bias == "promoted" else own[:1].clone()
    layer.bias = torch.nn.Parameter(new)
    y = layer(x)
    assert y.dtype == (base + new).dtype and torch.allclose(y, base + new, rtol=1e-4, atol=1e-4)
    y.abs().sum().backward()
    assert layer.bias.grad.shape == new.shape


@pytest.mark.parametrize("kind,planes", [("f32", 2), ("c64", 5), ("base4", 2)])
@pytest.mark.parametrize("save", [0, -1])
def test_what_a_layer_holds_for_its_backward(dev, kind, planes, save):
    """Between forward and backward a layer holds its input and, under the option's default, one plane per phase boundary
    (24 stages: three phases of 8 for floats, six of 4 for complex values) next to the re-ordered twiddles."""
    from conftest import abi_option
    layer = _layer(kind, 4096, 4096, dev, bias=False, nblocks=2)
    x = torch.randn(1024, 4096, dtype=torch.complex64 if kind == "c64" else torch.float32, device=dev)
    plane = x.numel() * x.element_size()
    with abi_option("autograd_save", save):
        layer(x)
        before = torch.cuda.memory_allocated()
        y = layer(x)
        held = torch.cuda.memory_allocated() - before - plane
        del y
        assert torch.cuda.memory_allocated() == before
    assert held < 4096 if save == 0 else planes * plane <= held < (planes + 0.5) * plane


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("make", [lambda s: s.circulant(torch.randn(12)), lambda s: s.circulant(torch.randn(16)), lambda s: s.fft(16),
                                  lambda s: s.ifft(16, br_first=False)], ids=["circulant12", "circulant16", "fft", "ifft"])
def test_pipelines_trace_and_vmap(dev, make):
    """Under a tracer or a functorch transform a pipeline runs its links, which have rules there."""
    from butterfly_b200 import special
    torch.manual_seed(8)
    f = make(special).to(dev)
    b = f[0].butterfly
    x = torch.randn(2, 5, b.in_size, dtype=torch.float32 if f[0].real_in else torch.complex64, device=dev)
    traced = torch.jit.trace(f, x, check_trace=False)
    other = torch.randn_like(x)
    close = lambda a, c: (a - c).abs().max() <= 1e-5 * c.abs().max()
    assert close(traced(other), f(other)) and close(torch.func.vmap(f)(x), f(x))
    with torch.no_grad():
        assert close(torch.func.vmap(f)(x), f(x))


@pytest.mark.parametrize("in_size,out_size", [(64, 64), (64, 128), (256, 256), (512, 1024)])
def test_bias_gradients_of_narrow_rows(dev, in_size, out_size):
    """Rows that share a tile row, stacks full: the bias gradient has one order there too, and is as close to the float64 sum
    as PyTorch's own (1.5 for another order of as many additions)."""
    torch.manual_seed(in_size)
    layer = _layer("f32", in_size, out_size, dev)
    batch = (1 << 21) // in_size + 3
    x, g = torch.randn(batch, in_size, device=dev), torch.randn(batch, out_size, device=dev)
    first, again = (torch.autograd.grad(layer(x), layer.bias, g)[0] for _ in range(2))
    want = g.double().sum(0)
    off = lambda s: ((s.double() - want).norm() / want.norm()).item()
    assert torch.equal(first, again) and off(first) <= 1.5 * off(g.sum(0))
