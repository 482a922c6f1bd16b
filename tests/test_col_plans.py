"""Which library plan a column transform is made from (the tables of the column kernel
only where it is used), against a library that records the calls."""
import pytest

from openvsip_b200 import Fftm, _lib, col, row, vsip


class _Library:
    def __init__(self):
        self.made = []

    def fcb_supported_cols(self, n):
        return int(n in (756, 4096, 8192))

    def fcb_plan_fftm(self, *args):
        self.made.append("rows")
        return 0

    def fcb_plan_fftm_cols(self, *args):
        self.made.append("columns")
        return 0

    def fcb_destroy(self, h):
        return 0


@pytest.mark.parametrize("n,count,axis,made", [(756, 4, col, "columns"), (4096, 129, col, "columns"), (4096, 128, col, "rows"),
                                               (8192, 1, col, "rows"), (1007, 300, col, "rows"), (756, 300, row, "rows")])
def test_column_tables_only_where_they_are_used(monkeypatch, n, count, axis, made):
    fake = _Library()
    monkeypatch.setattr(vsip, "lib", lambda: fake)
    monkeypatch.setattr(_lib, "lib", lambda: fake)
    f = Fftm(*((n, count) if axis == col else (count, n)), axis=axis)
    assert fake.made == [made] and f._col_kernel == (made == "columns")
