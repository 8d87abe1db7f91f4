"""ct_workspace_bytes counts everything a call's workspace holds: the wave's
slots, the LNO VJP's mat_bar partials (one nocc x nocc matrix per job of a wave),
the job energies and the orbit table."""
import pytest

from pyscfad_b200 import native


@pytest.mark.parametrize("o,v", [(5, 9), (16, 120)])
def test_workspace_bytes_count_the_lno_partials(o, v, monkeypatch):
    monkeypatch.setenv("CTB_MAX_WAVE", "10")
    slots, partials = 10 * 7 * o ** 3 * 8, 10 * o * o * 8
    assert native.lib().ct_workspace_bytes(o, v, 0, 1) == slots + partials + v * (v + 1) * (v + 2) // 6 * 8 + o ** 3 * 4
