"""The field-address array of the host binding: as many addresses as fields are given, null pointers
for the rest (which the library refuses or, where a call does not read them, ignores)."""
import pytest
import torch

import pmfmhd


@pytest.mark.parametrize("n", [0, 3, 8, 9])
def test_missing_fields_are_null_pointers(n):
    ts = [torch.zeros(4) for _ in range(n)]
    a = list(pmfmhd._p9(ts))
    assert a == [t.data_ptr() for t in ts] + [None] * (9 - n)


def test_too_many_fields_are_refused():
    with pytest.raises((ValueError, IndexError)):
        pmfmhd._p9([torch.zeros(4) for _ in range(10)])
