"""Host side of the fused module chains (glue.py): what they refuse before anything reaches a device, and how they are put
together.  Nothing is computed here."""
import pytest
import torch


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
