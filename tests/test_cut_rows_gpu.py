"""Rows that end inside a block of 32 columns on the packed-pair forward kernel."""
import pytest
import torch

from conftest import abi_option, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("in_size,out_size,nblocks,B", [
    (1000, 1000, 2, 1205), (516, 3000, 1, 70), (540, 512, 2, 1), (2044, 2044, 2, 33), (4092, 4096, 1, 77), (7996, 8192, 1, 9), (1028, 2048, 1, 5)])
def test_forward(oracle_mod, in_size, out_size, nblocks, B):
    import butterfly_b200 as bb
    dev = torch.device("cuda", 0)
    torch.manual_seed(in_size)
    layer = bb.Butterfly(in_size, out_size, nblocks=nblocks)
    x = torch.randn(B, in_size)
    xe = x.double().unsqueeze(1).expand(B, layer.nstacks, in_size).contiguous()
    want = oracle_mod.multiply_fw(layer.twiddle.detach().double(), xe, True).reshape(B, -1)[:, :out_size] + layer.bias.detach().double()
    layer = layer.to(dev)
    # a row that continues behind the layer's columns: what lies there must not be read
    wide = torch.full((B, in_size + 32), float("nan"), device=dev)
    wide[:, :in_size] = x.to(dev)
    with torch.no_grad():
        before = bb.abi.launch_count()
        y, y2 = layer(x.to(dev)), layer(wide[:, :in_size])
        launches = bb.abi.launch_count() - before
        with abi_option("fw2", 0):
            plain = layer(x.to(dev))
    assert launches == 4  # re-ordering and product, twice
    assert rel_err(y.cpu().double(), want) < 2e-5
    assert torch.equal(y, plain) and torch.equal(y, y2)  # the generic kernel multiplies and adds in the same order
    assert bb.abi.device_error() == 0
