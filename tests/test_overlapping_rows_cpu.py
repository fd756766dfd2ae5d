"""Rows that overlap (``unfold``, ``expand``) have no leading dimension: taken as
n rows of `width` elements they would be read past their end (no GPU; the helpers
look at strides alone)."""
import pytest
import torch

from tsm_benchmark_b200 import api


@pytest.mark.parametrize("x", [torch.arange(50.0).unfold(0, 8, 1), torch.arange(50.0).unfold(0, 8, 7),
                               torch.zeros(8).expand(20, 8), torch.zeros(1, 1).expand(20, 1),
                               torch.zeros(20).as_strided((10, 8), (0, 1))])
def test_overlapping_rows_have_no_leading_dimension(x):
    with pytest.raises(ValueError, match="overlap"):
        api._ld(x)


@pytest.mark.parametrize("x,ld", [(torch.zeros(20, 8), 8), (torch.zeros(20, 8)[:, 2:5], 8), (torch.zeros(20, 8)[::3], 24),
                                  (torch.zeros(1, 8).expand(1, 8), 8), (torch.zeros(0, 8), 8), (torch.zeros(5, 1), 1),
                                  (torch.arange(48.0).unfold(0, 8, 8), 8), (torch.zeros(1, 5).t(), 1)])
def test_other_rows_keep_theirs(x, ld):
    assert api._ld(x) == ld


def test_autograd_copies_them():
    from tsm_benchmark_b200.autograd import _row_major
    assert _row_major(torch.zeros(20, 8)) and _row_major(torch.zeros(20, 8)[:, 2:5]) and _row_major(torch.zeros(1, 8))
    assert not _row_major(torch.zeros(8).expand(20, 8)) and not _row_major(torch.arange(50.0).unfold(0, 8, 1))
    assert not _row_major(torch.zeros(8, 20).t())
