"""A t3 handed to the iterative (T) solver is only read, also when it is the array
an earlier call returned (a view of the solver's own layout)."""
import pytest
import torch

from pyscfad_b200 import synth
from pyscfad_b200.cc import ccsd_t_iter
from test_oracle import _perturbed_fock

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(6, 9), (21, 3)])   # one step kernel, and a GEMM with the update kernel
def test_restart_leaves_t3_alone(o, v, cuda_dev):
    s = _perturbed_fock(synth.make_system(o, v, 3 * v, 3, fvo_sigma=0.02), 0.02, 7)
    conv, _, t3 = ccsd_t_iter.iterative_kernel(None, s, s.t1, s.t2, max_cycle=2)
    assert not conv
    kept = t3.clone()
    for cycles in (1, 2, 3):
        _, _, new = ccsd_t_iter.iterative_kernel(None, s, s.t1, s.t2, t3=t3, max_cycle=cycles)
        assert torch.equal(t3, kept)
        assert not torch.equal(new, kept)
