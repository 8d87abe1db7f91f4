"""The names the LNO timing prints for the profile kinds follow the path taken."""
import pytest

from pyscfad_b200.lno.timing import kind_names


@pytest.mark.parametrize("mode,nocc,cube", [("fp64", 2, True), ("fp64", 24, True), ("fp64", 1, False),
                                            ("fp64", 25, False), ("tf32", 16, False)])
def test_kind_names(mode, nocc, cube):
    names = kind_names(mode, nocc)
    assert ("job kernel" in names[0] and "job kernel" in names[4]) is cube
    # F2 as a pass of its own is the mixed path's (kind 13) alone
    assert 1 not in names
    assert set(names) == {0, *range(2, 16)}
