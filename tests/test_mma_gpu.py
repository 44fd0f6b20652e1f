"""Products as tensor-core passes (option "mma" = 1) against float64: tiles with few and missing rows, cut and padded columns,
rows between alignments, several stacks, windows at every place of a row, both directions, both dtypes, both radices."""
import pytest
import torch

from conftest import abi_option

pytestmark = pytest.mark.gpu

# A pass rounds its sums to 2^-24 four times and its result once, and drops what is below 2^-24 of a product: 1.2e-7 at most on
# average over the columns, five passes at most; the operator gradient adds float32 sums over 128 rows at a time.
TOL = 6e-7
TOL_GRAD = 1.2e-6


@pytest.fixture(scope="module")
def dev():
    return torch.device("cuda", 0)


def rel2(a, b):
    a, b = a.detach().cpu().to(b.dtype), b.detach()
    return ((a - b).norm() / b.norm()).item()


@pytest.mark.parametrize("cplx,log_n,nblocks,S,B,inc", [
    (False, 6, 2, 1, 1, True), (False, 6, 2, 2, 129, False), (False, 7, 2, 3, 128, True), (False, 9, 1, 1, 127, True),
    (False, 10, 1, 2, 300, False), (False, 10, 2, 4, 257, True), (False, 11, 2, 1, 130, False), (False, 12, 2, 1, 300, True),
    (False, 13, 1, 1, 200, True), (False, 14, 1, 1, 65, False),
    (True, 5, 2, 2, 300, True), (True, 6, 2, 1, 129, False), (True, 9, 1, 2, 128, True), (True, 10, 2, 1, 257, True),
    (True, 11, 1, 1, 300, True), (True, 12, 1, 1, 70, False)])
@pytest.mark.parametrize("save", [0, 1])
def test_multiply(dev, oracle_mod, cplx, log_n, nblocks, S, B, inc, save):
    import butterfly_b200 as bb
    n, dt, wide = 1 << log_n, torch.complex64 if cplx else torch.float32, torch.complex128 if cplx else torch.float64
    torch.manual_seed(log_n + B)
    tw = torch.randn(S, nblocks, log_n, n // 2, 2, 2, dtype=dt) / 2 ** 0.5
    x, g = torch.randn(B, S, n, dtype=dt), torch.randn(B, S, n, dtype=dt)
    want_y = oracle_mod.multiply_fw(tw.to(wide), x.to(wide), inc)
    want_d, want_dx = oracle_mod.multiply_bw(tw.to(wide), x.to(wide), g.to(wide), inc)
    with abi_option("mma", 1), abi_option("autograd_save", save):
        t, xd = tw.to(dev).requires_grad_(True), x.to(dev).requires_grad_(True)
        y = bb.butterfly_multiply(t, xd, inc)
        d, dx = torch.autograd.grad(y, [t, xd], g.to(dev))
        d2, dx2 = bb.butterfly_multiply_bw(t.detach(), xd.detach(), g.to(dev), inc)
    assert rel2(y, want_y) < TOL and rel2(dx, want_dx) < TOL and rel2(d, want_d) < TOL_GRAD
    assert torch.equal(dx, dx2) and torch.equal(d, d2)  # the same bits with activations kept and made again
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("kind,in_size,out_size,nblocks,B", [
    ("f32", 1000, 3000, 2, 150), ("f32", 1023, 1021, 2, 129), ("f32", 1024, 4096, 2, 200), ("f32", 70, 100, 2, 300),
    ("f32", 4090, 4100, 1, 130), ("c64", 61, 64, 2, 300), ("c64", 500, 700, 2, 129), ("c64", 1999, 2000, 1, 40),
    ("base4", 64, 64, 2, 129), ("base4", 1000, 2000, 2, 200), ("base4", 4096, 4000, 1, 100), ("base4", 500, 512, 2, 64)])
@pytest.mark.parametrize("save", [0, 1])
def test_layer(dev, oracle_mod, kind, in_size, out_size, nblocks, B, save):
    import butterfly_b200 as bb
    torch.manual_seed(in_size)
    layer = (bb.ButterflyBase4 if kind == "base4" else bb.Butterfly)(in_size, out_size, bias=True, complex=kind == "c64", nblocks=nblocks)
    dt, wide = (torch.complex64, torch.complex128) if kind == "c64" else (torch.float32, torch.float64)
    x, g = torch.randn(B, in_size, dtype=dt), torch.randn(B, out_size, dtype=dt)
    S, n = layer.nstacks, layer.n
    xe = x.to(wide).unsqueeze(1).expand(B, S, in_size).contiguous()
    gp = torch.zeros(B, S * n, dtype=wide)
    gp[:, :out_size] = g
    gp = gp.view(B, S, n)
    if kind == "base4":
        tws = [layer.twiddle4.detach().to(wide), layer.twiddle2.detach().to(wide)]
        y = oracle_mod.base4_fw(*tws, xe, True)
        *dtw, dx = oracle_mod.base4_bw(*tws, xe, gp, True)
    else:
        tws = [layer.twiddle.detach().to(wide)]
        y = oracle_mod.multiply_fw(*tws, xe, True)
        *dtw, dx = oracle_mod.multiply_bw(*tws, xe, gp, True)
    want = [y.reshape(B, S * n)[:, :out_size] + layer.bias.detach().to(wide), dx.sum(1), g.to(wide).sum(0), *dtw]
    layer = layer.to(dev)
    params = [layer.twiddle4, layer.twiddle2] if kind == "base4" else [layer.twiddle]
    xd = x.to(dev).requires_grad_(True)
    with abi_option("mma", 1), abi_option("autograd_save", save):
        out = layer(xd)
        grads = torch.autograd.grad(out, [xd, layer.bias] + params, g.to(dev))
    for got, ref, what in zip([out, *grads], want, ("output", "d_input", "d_bias", "d_twiddle", "d_twiddle2")):
        if ref.numel():
            assert rel2(got, ref) < (TOL if what in ("output", "d_input") else TOL_GRAD), what
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("pitch,offset", [(70, 0), (68, 4), (67, 1), (66, 2)])
def test_strided_rows(dev, oracle_mod, pitch, offset):
    import butterfly_b200 as bb
    torch.manual_seed(pitch)
    tw = torch.randn(1, 2, 6, 32, 2, 2) / 2 ** 0.5
    rows, g = torch.randn(130, pitch, device=dev)[:, offset:offset + 64].unsqueeze(1), torch.randn(130, 1, 64)
    want_d, want_dx = oracle_mod.multiply_bw(tw.double(), rows.cpu().double(), g.double(), True)
    with abi_option("mma", 1):
        d, dx = bb.butterfly_multiply_bw(tw.to(dev), rows, g.to(dev), True)
    assert rel2(dx, want_dx) < TOL and rel2(d, want_d) < TOL_GRAD


def _same(got, want, exact):
    """Infinities with their signs and NaN in the same places; the rest bit for bit, or to what the order of a sum over 300
    rows (the phases have none that is fixed) may change, 300 2^-24 of it."""
    for a, b, e in zip(got, want, exact):
        a, b = (torch.view_as_real(t) if t.is_complex() else t for t in (a.detach(), b.detach()))
        scale = b[torch.isfinite(b)].double().pow(2).mean().sqrt().item() if torch.isfinite(b).any() else 0.0
        torch.testing.assert_close(a.double(), b.double(), rtol=0 if e else 2e-5, atol=0 if e else 2e-5 * scale, equal_nan=True)


@pytest.mark.parametrize("cplx,log_n,inc", [(False, 10, True), (False, 7, False), (True, 8, True)])
@pytest.mark.parametrize("factors", ["normal", "identity", "positive"])
@pytest.mark.parametrize("place,value", [("x", float("inf")), ("x", float("-inf")), ("x", float("nan")), ("x", -3.4e38), ("x", 1.2e12),
                                         ("grad", float("inf")), ("grad", float("nan")), ("grad", 3e38), ("twiddle", float("inf")),
                                         ("twiddle", float("nan")), ("twiddle", 1e30), ("sums", 1e12)])
@pytest.mark.parametrize("save", [0, 1])
def test_values_that_are_not_ordinary_give_what_the_phases_give(dev, cplx, log_n, inc, factors, place, value, save):
    """A stage multiplies zeros by infinities and overflows halfway; an operator that stands for several stages does not."""
    import butterfly_b200 as bb
    n, B, dt = 1 << log_n, 300, torch.complex64 if cplx else torch.float32
    torch.manual_seed(3)
    tw = torch.randn(1, 2, log_n, n // 2, 2, 2, dtype=dt, device=dev) / 2 ** 0.5
    if factors == "identity":
        tw = torch.eye(2, dtype=dt, device=dev).expand_as(tw).contiguous()
    elif factors == "positive":
        tw = tw.abs().to(dt) / 8
    x, g = (torch.randn(B, 1, n, dtype=dt, device=dev) for _ in range(2))
    if place == "sums":
        x, g = (torch.rand(B, 1, n, device=dev).to(dt) * value for _ in range(2))
    else:
        {"x": x, "grad": g, "twiddle": tw}[place].view(-1)[n + 9 if place != "twiddle" else 5] = value
    res = []
    for mma in (0, 1):
        with abi_option("mma", mma), abi_option("autograd_save", save):
            t, xd = tw.clone().requires_grad_(True), x.clone().requires_grad_(True)
            y = bb.butterfly_multiply(t, xd, inc)
            d, dx = torch.autograd.grad(y, [t, xd], g)
            res.append([y, dx, d])
    _same(res[1], res[0], (place in ("x", "twiddle"), place != "sums", False))  # (a forward does not know of the gradient)
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("kind,in_size,out_size", [("f32", 1000, 3000), ("f32", 1024, 4096), ("c64", 500, 700), ("base4", 1000, 1000), ("base4", 16384, 16384)])
@pytest.mark.parametrize("place", ["x", "grad", "twiddle"])
@pytest.mark.parametrize("save", [0, 1])
def test_layers_of_values_that_are_not_ordinary(dev, kind, in_size, out_size, place, save):
    import butterfly_b200 as bb
    torch.manual_seed(4)
    layer = (bb.ButterflyBase4 if kind == "base4" else bb.Butterfly)(in_size, out_size, bias=True, complex=kind == "c64", nblocks=2).to(dev)
    dt = torch.complex64 if kind == "c64" else torch.float32
    x, g = torch.randn(150, in_size, dtype=dt, device=dev), torch.randn(150, out_size, dtype=dt, device=dev)
    params = sorted((p for p in layer.parameters() if p.numel()), key=lambda p: -p.numel())
    {"x": x, "grad": g, "twiddle": params[0].data}[place].view(-1)[in_size + 9] = float("-inf")
    res = []
    for mma in (0, 1):
        xd = x.clone().requires_grad_(True)
        with abi_option("mma", mma), abi_option("autograd_save", save):
            out = layer(xd)
            res.append([out, *torch.autograd.grad(out, [xd] + params, g)])
    _same(res[1], res[0], [place != "grad", layer.nstacks == 1] + [False] * len(params))
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("cplx,log_n", [(False, 6), (False, 10), (True, 9)])
@pytest.mark.parametrize("what", ["rows", "gradients", "both", "factors", "subnormal rows"])
def test_small_values_keep_24_bits(dev, oracle_mod, cplx, log_n, what):
    """Down to the end of float32's range: slices and operators are scaled, so that their last parts stay normal numbers."""
    import butterfly_b200 as bb
    n, B = 1 << log_n, 300
    dt, wide = (torch.complex64, torch.complex128) if cplx else (torch.float32, torch.float64)
    torch.manual_seed(log_n)
    tw = torch.randn(1, 2, log_n, n // 2, 2, 2, dtype=dt) / 2 ** 0.5
    x, g = torch.randn(B, 1, n, dtype=dt), torch.randn(B, 1, n, dtype=dt)
    if what == "factors":  # operators of 2^-108
        tw = tw / 2 ** (108 // (2 * log_n))
    elif what == "subnormal rows":
        tw = torch.eye(2, dtype=dt).expand_as(tw).contiguous()
        x, g = x * 2.0 ** -131, g * 2.0 ** -131
    else:
        x = x * (2.0 ** -115 if what == "rows" else 2.0 ** -55 if what == "both" else 1)
        g = g * (2.0 ** -115 if what == "gradients" else 2.0 ** -55 if what == "both" else 1)
    want_y = oracle_mod.multiply_fw(tw.to(wide), x.to(wide), True)
    want_d, want_dx = oracle_mod.multiply_bw(tw.to(wide), x.to(wide), g.to(wide), True)
    with abi_option("mma", 1):
        t, xd = tw.to(dev).requires_grad_(True), x.to(dev).requires_grad_(True)
        y = bb.butterfly_multiply(t, xd, True)
        d, dx = torch.autograd.grad(y, [t, xd], g.to(dev))
    if what == "subnormal rows":
        assert torch.equal(y.detach().cpu(), x) and torch.equal(dx.cpu(), g)  # (products of two such values are below the range)
    else:
        assert rel2(y, want_y) < TOL and rel2(dx, want_dx) < TOL and rel2(d, want_d) < TOL_GRAD


def test_the_largest_ordinary_values_stay_on_the_passes(dev, oracle_mod):
    """Rows below 2^40 and operators below 2^20, whatever the phases make of them."""
    import butterfly_b200 as bb
    torch.manual_seed(5)
    tw = torch.randn(1, 2, 6, 32, 2, 2) / 2 ** 0.5
    x, g = torch.randn(300, 1, 64) * 2.0 ** 36, torch.randn(300, 1, 64) * 2.0 ** 20
    want_y = oracle_mod.multiply_fw(tw.double(), x.double(), True)
    want_d, want_dx = oracle_mod.multiply_bw(tw.double(), x.double(), g.double(), True)
    with abi_option("mma", 1):
        t, xd = tw.to(dev).requires_grad_(True), x.to(dev).requires_grad_(True)
        y = bb.butterfly_multiply(t, xd, True)
        d, dx = torch.autograd.grad(y, [t, xd], g.to(dev))
    assert rel2(y, want_y) < TOL and rel2(dx, want_dx) < TOL and rel2(d, want_d) < TOL_GRAD


@pytest.mark.parametrize("cplx,log_n,B", [(False, 12, 16384), (True, 10, 4096)])
@pytest.mark.parametrize("inc", [True, False])
def test_large_training_steps_under_the_default_rule(dev, cplx, log_n, B, inc):
    """Two blocks: one direction runs as passes, the other, which is cut into more groups, on the phases.  Both train, and agree
    with the phases to what two float32 evaluations of 24 factors may differ by."""
    import butterfly_b200 as bb
    n, dt = 1 << log_n, torch.complex64 if cplx else torch.float32
    torch.manual_seed(log_n)
    tw = (torch.randn(1, 2, log_n, n // 2, 2, 2, dtype=dt, device=dev) / 2 ** 0.5).requires_grad_(True)
    x, g = (torch.randn(B, 1, n, dtype=dt, device=dev) for _ in range(2))
    x.requires_grad_(True)
    got, passes = [], []
    for mma in (-1, 0):
        with abi_option("mma", mma):
            bb.abi.profile_enable()
            y = bb.butterfly_multiply(tw, x, inc)
            got.append([y.detach()] + list(torch.autograd.grad(y, [tw, x], g)))
            passes.append(sum(n for k, (n, _) in bb.abi.profile_collect().items() if "mma" in k))
            bb.abi.profile_enable(False)
    assert (passes[0] > 0) == inc and passes[1] == 0
    for a, b in zip(*got):
        assert ((a - b).norm() / b.norm()).item() < 2e-6
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("cplx,log_n", [(False, 6), (False, 7), (True, 5)])
@pytest.mark.parametrize("positive", [False, True])
def test_many_tiles_to_a_cta(dev, oracle_mod, cplx, log_n, positive):
    """700001 rows of one or two windows: 37 to 74 tiles of a block to every CTA, so that the sums that run on over tiles are
    taken out on the way and at the end, and the barriers go through many turns.  Sums of one sign: what the accumulators cut
    adds up, by half a unit of the last place for each of the four instructions of a short sum and as much again for rows,
    gradients and the sums that run on.  A product of n columns is an n x n matrix:
    its gradient, made in float64, goes through the oracle."""
    import butterfly_b200 as bb
    n, B = 1 << log_n, 700001
    dt, wide = (torch.complex64, torch.complex128) if cplx else (torch.float32, torch.float64)
    torch.manual_seed(log_n)
    tw = torch.randn(1, 2, log_n, n // 2, 2, 2, dtype=dt) / 2 ** 0.5
    x, g = (torch.randn(B, 1, n, dtype=dt, device=dev) for _ in range(2))
    if positive:
        tw, x, g = (v.abs().to(dt) for v in (tw, x, g))
    with abi_option("mma", 1):
        t, xd = tw.to(dev).requires_grad_(True), x.requires_grad_(True)
        y = bb.butterfly_multiply(t, xd, True)
        d, dx = torch.autograd.grad(y, [t, xd], g)
    eye = torch.eye(n, dtype=wide).unsqueeze(1)
    m = oracle_mod.multiply_fw(tw.to(wide), eye, True)[:, 0]  # row i: the product's i-th column
    xw, gw = x.detach()[:, 0].to(wide), g[:, 0].to(wide)
    want_d, _ = oracle_mod.multiply_bw(tw.to(wide), eye, (xw.conj().T @ gw).cpu().unsqueeze(1), True)
    md = m.to(dev)
    for got, want in ((y[:, 0], xw @ md), (dx[:, 0], gw @ md.conj().T)):
        assert ((got.detach().to(wide) - want).norm() / want.norm()).item() < TOL
    assert rel2(d, want_d) < (4 * 2 ** -25 + 2 * 2 ** -25 if positive else TOL_GRAD)
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("kind", ["multiply", "layer", "base4"])
@pytest.mark.parametrize("first,then", [(1, 0), (0, 1)])
def test_an_option_set_between_forward_and_backward(dev, kind, first, then):
    """What the forward saved is laid out for the passes or for the phases; a backward after the switch does not read it."""
    import butterfly_b200 as bb
    torch.manual_seed(6)
    if kind == "multiply":
        tw = (torch.randn(1, 2, 9, 256, 2, 2, device=dev) / 2 ** 0.5).requires_grad_(True)
        f, params = lambda r: bb.butterfly_multiply(tw, r, True), [tw]
    else:
        f = (bb.ButterflyBase4 if kind == "base4" else bb.Butterfly)(512, 512, bias=False, nblocks=2).to(dev)
        params = [p for p in f.parameters() if p.numel()]
    x = torch.randn(300, *((1,) if kind == "multiply" else ()), 512, device=dev, requires_grad=True)
    g = torch.randn_like(x)
    res = []
    for a, b in ((first, then), (0, 0)):
        with abi_option("autograd_save", 1):
            with abi_option("mma", a):
                y = f(x)
            with abi_option("mma", b):
                res.append(torch.autograd.grad(y, [x] + params, g))
    for a, b in zip(*res):
        assert ((a - b).norm() / b.norm()).item() < 2 * TOL_GRAD
    assert bb.abi.device_error() == 0


@pytest.mark.parametrize("cplx", [False, True])
def test_the_pair_of_one_buffer_stays_on_the_phases(dev, cplx):
    """bfly_fw_*_saving and bfly_bw_*_saved have no work space for the passes, wherever these would run."""
    from butterfly_b200 import abi
    dt = torch.complex64 if cplx else torch.float32
    torch.manual_seed(2)
    tw = torch.randn(1, 2, 10, 512, 2, 2, dtype=dt, device=dev) / 2 ** 0.5
    x, g = (torch.randn(300, 1, 1024, dtype=dt, device=dev) for _ in range(2))
    with abi_option("mma", 1):
        out, snaps, rc = abi.fw_saving(tw, x, True, check=False)
        assert rc == 0
        d, dx, rc = abi.bw_saved(tw, x, g, snaps, True, check=False)
        assert rc == 0
    with abi_option("mma", 0):
        want, want_x, _ = abi.bw(tw, x, g, True)
    assert torch.equal(dx, want_x) and ((d - want).norm() / want.norm()).item() < 1e-6


def _factors(kind, shape, dt):
    """Twiddles, and rows or gradients to go with them."""
    B, (nb, log_n, half) = 300, shape
    tw, (x, g) = torch.randn(1, nb, log_n, half, 2, 2, dtype=dt) / 2 ** 0.5, torch.randn(2, B, 1, 2 * half, dtype=dt)
    eye = torch.eye(2, dtype=dt).expand_as(tw)
    if kind == "positive":
        tw, x, g = (t.abs().to(dt) for t in (tw, x, g))
    elif kind == "uniform":
        tw, x, g = (torch.rand(t.shape).to(dt) for t in (tw, x, g))
    elif kind == "one-hot rows":
        x, g = (t * torch.nn.functional.one_hot(torch.randint(0, 2 * half, (B, 1)), 2 * half) for t in (x, g))
    elif kind == "sparse rows":
        x, g = (t * (torch.rand(t.shape) < 0.01) for t in (x, g))
    elif kind == "near the identity":
        tw = eye + 1e-3 * tw
    elif kind == "averages":
        tw, x, g = torch.full_like(tw, 0.5), x.abs().to(dt), g.abs().to(dt)
    elif kind == "identity":
        tw = eye
    elif kind == "permutation":
        tw = torch.where(torch.rand(1, nb, log_n, half, 1, 1) < 0.5, eye, eye.flip(-1))
    elif kind == "powers of two":
        tw = eye * 2.0 ** torch.randint(-2, 3, (1, nb, log_n, half, 1, 2)) * torch.where(torch.rand(1, nb, log_n, half, 1, 2) < 0.5, 1.0, -1.0)
    return tw.contiguous(), x, g


@pytest.mark.parametrize("cplx,log_n,nblocks,inc", [(False, 10, 2, True), (False, 10, 1, True), (False, 9, 2, False), (True, 8, 2, True)])
@pytest.mark.parametrize("kind", ["normal", "positive", "uniform", "one-hot rows", "sparse rows", "near the identity", "averages", "identity",
                                  "permutation", "powers of two"])
def test_no_further_from_float64_than_the_phases(dev, oracle_mod, kind, cplx, log_n, nblocks, inc):
    """Whatever the distribution.  A pass rounds each result once where the phases round once per factor; factors that only
    move and scale columns give every bit back.  Gradients of the factors, sums over the rows, have a bound of their own: the
    tensor cores' accumulators cut four times, half of 2^-23 each, and rows and gradients carry the error of up to three passes."""
    import butterfly_b200 as bb
    dt, wide = (torch.complex64, torch.complex128) if cplx else (torch.float32, torch.float64)
    torch.manual_seed(log_n + nblocks)
    tw, x, g = _factors(kind, (nblocks, log_n, 1 << (log_n - 1)), dt)
    want_y = oracle_mod.multiply_fw(tw.to(wide), x.to(wide), inc)
    want_d, want_dx = oracle_mod.multiply_bw(tw.to(wide), x.to(wide), g.to(wide), inc)
    err = []
    for mma in (0, 1):
        with abi_option("mma", mma), abi_option("autograd_save", 1):
            t, xd = tw.to(dev).requires_grad_(True), x.to(dev).requires_grad_(True)
            y = bb.butterfly_multiply(t, xd, inc)
            d, dx = torch.autograd.grad(y, [t, xd], g.to(dev))
        err.append([rel2(y, want_y), rel2(dx, want_dx), rel2(d, want_d)])
    phases, passes = err
    assert passes[0] <= phases[0] and passes[1] <= phases[1] and passes[2] < 4 * 2 ** -24 + 3 * 2 ** -24
    if kind in ("identity", "permutation", "powers of two"):
        assert passes[:2] == [0.0, 0.0]


def test_threads_with_products_of_different_groups(dev):
    """Launches of one kernel with different amounts of shared memory, from two host threads on streams of their own."""
    import threading
    import butterfly_b200 as bb
    torch.manual_seed(8)
    jobs = []
    for log_n, nblocks in ((6, 2), (10, 1)):  # groups of twelve factors, and of five
        tw = torch.randn(1, nblocks, log_n, 1 << (log_n - 1), 2, 2, device=dev) / 2 ** 0.5
        x, g = (torch.randn(200, 1, 1 << log_n, device=dev) for _ in range(2))
        jobs.append((tw, x, g))
    got, errors = [[], []], []
    with abi_option("mma", 1):
        want = [bb.butterfly_multiply_bw(*j, True) for j in jobs]
        torch.cuda.synchronize()

        def work(k):
            try:
                with torch.cuda.stream(torch.cuda.Stream(dev)):
                    for _ in range(200):
                        got[k] = bb.butterfly_multiply_bw(*jobs[k], True)
                    torch.cuda.current_stream().synchronize()
            except Exception as e:  # (a refused launch)
                errors.append(e)
        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not errors
    for a, b in zip(want, got):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_captured_training_steps_look_at_the_values_of_each_replay(dev):
    import butterfly_b200 as bb
    torch.manual_seed(9)
    tw = (torch.randn(1, 2, 9, 256, 2, 2, device=dev) / 2 ** 0.5).requires_grad_(True)
    x, g = torch.randn(300, 1, 512, device=dev, requires_grad=True), torch.randn(300, 1, 512, device=dev)

    def step():
        y = bb.butterfly_multiply(tw, x, True)
        return [y.detach()] + list(torch.autograd.grad(y, [x, tw], g))
    with abi_option("mma", 1):
        side = torch.cuda.Stream(dev)
        with torch.cuda.stream(side):
            step()
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = step()
        for value in (1.0, float("inf"), 2.0, float("nan"), 3.0):
            with torch.no_grad():
                x.view(-1)[5] = value
            graph.replay()
            _same(outs, step(), (True, True, False))
    assert bb.abi.device_error() == 0
