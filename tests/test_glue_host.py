"""Host side of the fused module chains (glue.py): what they refuse before anything reaches a device, and how they are put
together.  Nothing is computed here."""
import pytest
import torch
from torch import nn


@pytest.mark.parametrize("br_first", [True, False])
@pytest.mark.parametrize("width", [1, 5, 7, 9, 16])
def test_pipelines_of_whole_rows_refuse_other_widths(br_first, width):
    """A gather over a row shorter than its permutation would read past the row: refused on the host, as the link-by-link
    reshape did."""
    from butterfly_b200 import special
    f = special.fft(8, br_first=br_first)
    with pytest.raises(RuntimeError, match="rows of 8 entries"):
        f(torch.randn(3, width, dtype=torch.complex64))


def test_glue_operator_refuses_gathers_of_short_rows():
    import butterfly_b200 as bb
    tw = torch.randn(1, 1, 3, 4, 2, 2)
    with pytest.raises(RuntimeError, match="in_perm needs rows of 8 entries"):
        bb.butterfly_multiply_glue(tw, torch.randn(2, 1, 7), True, in_perm=torch.randperm(8, dtype=torch.int32))


def test_a_lone_butterfly_of_cut_rows_stays_a_butterfly():
    """Nothing to fold into its launch: the layer itself, with its methods and its state's names."""
    import butterfly_b200 as bb
    from butterfly_b200 import special
    c = special.circulant(torch.randn(12, dtype=torch.complex64), separate_diagonal=False)
    assert type(c) is bb.Butterfly and list(c.state_dict()) == ["twiddle"]
    whole = special.circulant(torch.randn(16, dtype=torch.complex64), separate_diagonal=False)
    assert isinstance(whole, bb.glue.ButterflyPipeline)


@pytest.mark.parametrize("n", [12, 16])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("separate_diagonal", [False, True])
def test_state_of_the_link_by_link_form_loads(n, cplx, separate_diagonal):
    """Checkpoints of circulants written before their lengths were fused (and of fused=False modules) keep loading."""
    from butterfly_b200 import special
    if n == 16 and cplx and not separate_diagonal:
        pytest.skip("the unfused form is one Butterfly, whose state carries no link names")
    col = lambda: torch.randn(n, dtype=torch.complex64 if cplx else torch.float32)
    chained = special.circulant(col(), separate_diagonal=separate_diagonal, fused=False)
    fused = special.circulant(col(), separate_diagonal=separate_diagonal)
    want = [p.detach().clone() for p in chained.parameters()]
    fused.load_state_dict(chained.state_dict())
    assert all(torch.equal(a, b) for a, b in zip(fused.parameters(), want))
    again = special.circulant(col(), separate_diagonal=separate_diagonal)
    again.load_state_dict(fused.state_dict())  # its own form, too
    assert all(torch.equal(a, b) for a, b in zip(again.parameters(), want))
    holder = nn.ModuleDict({"a": special.circulant(col(), separate_diagonal=separate_diagonal)})
    holder.load_state_dict({"a." + k: v for k, v in chained.state_dict().items()})
    assert all(torch.equal(a, b) for a, b in zip(holder.parameters(), want))


def test_state_of_a_chain_with_kept_links_loads():
    import copy

    import butterfly_b200 as bb
    from butterfly_b200 import glue
    from butterfly_b200.permutation import FixedPermutation
    links = lambda: [nn.Linear(8, 8), FixedPermutation(torch.randperm(8)), bb.Butterfly(8, 8, False), nn.Linear(8, 8),
                     bb.Butterfly(8, 8, False), FixedPermutation(torch.randperm(8))]
    chain, fused = nn.Sequential(*links()), glue.fuse(nn.Sequential(*links()))
    assert len(fused) == 4
    state = {k: v.clone() for k, v in chain.state_dict().items()}
    copy.deepcopy(fused).load_state_dict(state)
    fused.load_state_dict(state)
    for (_, p), q in zip(chain.named_parameters(), fused.parameters()):
        assert torch.equal(p, q)
    assert torch.equal(fused[1].in_perm.long(), chain[1].permutation) and torch.equal(fused[3].out_perm.long(), chain[5].permutation)
    assert len(fused[:2]) == 2
    with pytest.raises(RuntimeError, match="Missing key"):
        fused.load_state_dict({k: v for k, v in state.items() if not k.startswith("2.")})
