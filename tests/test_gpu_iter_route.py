"""Which kernel forms a step of the iterative (T) solver: one kernel where it is
the faster one, else a GEMM on an occupied-major copy and the update kernel
(one kernel at every size took 21 times the time of the two at nocc=64/nvir=6).
Both against the numpy solver at the tolerances of test_gpu_iter.py: energies
within 1e-11 relative, amplitudes within 1e-9 of their largest element."""

import numpy as np
import pytest

from oracle import ccsd_t_iter_np as it
from pyscfad_b200 import native, synth
from pyscfad_b200.cc import ccsd_t_iter
from test_oracle import _perturbed_fock


@pytest.mark.parametrize("o,v,one", [(1, 300, True), (8, 40, True), (9, 200, True), (20, 60, True), (11, 27, True),
                                     (19, 9, True), (11, 60, False), (13, 28, False), (19, 10, False), (21, 1, False),
                                     (22, 4, False), (24, 16, False), (64, 6, False)])
def test_step_rule(o, v, one):
    assert ccsd_t_iter._one_kernel_step(o, v) is one


class _Spy:
    """The library with the names of the called t3 entries kept."""

    def __init__(self, lib):
        self._lib, self.calls = lib, set()

    def __getattr__(self, name):
        if name.startswith("ct_t3_"):
            self.calls.add(name)
        return getattr(self._lib, name)


@pytest.mark.gpu
@pytest.mark.parametrize("o,v,entry", [(8, 6, "ct_t3_step"), (11, 5, "ct_t3_step"), (21, 3, "ct_t3_update"),
                                       (22, 2, "ct_t3_update"), (33, 2, "ct_t3_update")])
def test_solver_on_both_routes(o, v, entry, cuda_dev, monkeypatch):
    s = _perturbed_fock(synth.make_system(o, v, 3 * v, 3, fvo_sigma=0.02), 0.02, 7)
    spy = _Spy(native.lib())
    monkeypatch.setattr(native, "lib", lambda: spy)
    conv_r, e_r, t3_r, hist = it.iterative_kernel(s.t1, s.t2, s.mo_energy, s.fock, s.ovov, s.ovoo, s.ovvv,
                                                  tol=1e-12, tolnormt=1e-11)
    conv, e, t3 = ccsd_t_iter.iterative_kernel(None, s, s.t1, s.t2, tol=1e-12, tolnormt=1e-11)
    assert spy.calls == {"ct_t3_init", entry}
    assert conv and conv_r and len(hist) > 3
    assert abs(e - e_r) <= 1e-11 * abs(e_r), (e, e_r)
    assert np.abs(t3.cpu().numpy() - t3_r).max() <= 1e-9 * np.abs(t3_r).max()
