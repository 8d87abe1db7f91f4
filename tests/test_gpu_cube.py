"""The float64 path that keeps a job's cube in shared memory (nocc 2-24)
against the numpy oracle, at the edges of its tiles: every count of 8-row
tiles over the 2 nocc rows, one and several column passes, one and several
K chunks of 48 virtuals, and the slot path's sizes on both sides of it.

Tolerances: the repository's float64 ones (energies 1e-12 relative, gradients
1e-10 of each gradient's norm)."""
import math

import numpy as np
import pytest
import torch

from oracle import ccsd_t_np as onp
from pyscfad_b200 import surrogate, synth, triples

pytestmark = pytest.mark.gpu
KEYS = ("mo_energy", "t1T", "t2T", "vooo", "fvo", "vvop")


def _system(o, v, fvo, seed=5):
    return synth.reference_layouts(synth.make_system(o, v, 3 * v, seed, fvo_sigma=fvo))


def _dev(L, dev):
    return {k: torch.from_numpy(np.ascontiguousarray(x)).to(dev) for k, x in L.items()}


@pytest.mark.parametrize("o,v,fvo", [(1, 6, 0.02), (2, 6, 0.02), (3, 5, 0.0), (4, 50, 0.02), (5, 7, 0.02), (8, 9, 0.0),
                                     (9, 11, 0.02), (12, 8, 0.0), (13, 7, 0.02), (16, 17, 0.02), (17, 6, 0.0),
                                     (19, 8, 0.02), (20, 7, 0.0), (21, 6, 0.02), (23, 9, 0.02), (24, 8, 0.02),
                                     (25, 6, 0.02), (6, 1, 0.02)])
def test_vjp_matches_oracle(o, v, fvo, cuda_dev):
    L = _system(o, v, fvo)
    e_ref, g_ref = onp.energy_vjp(L, 1.0)
    e, g = triples.energy_vjp(_dev(L, cuda_dev), 2.0)
    assert abs(e.item() - e_ref) <= 1e-12 * abs(e_ref) + 1e-14
    assert abs(triples.energy(_dev(L, cuda_dev)).item() - e_ref) <= 1e-12 * abs(e_ref) + 1e-14
    for k in KEYS:
        err = np.linalg.norm(g[k].cpu().numpy() - g_ref[k])
        assert err <= 1e-10 * np.linalg.norm(g_ref[k]) + 1e-15, (k, err)


@pytest.mark.parametrize("o,v", [(3, 47), (10, 49), (14, 97), (17, 60), (20, 52), (23, 61), (24, 97)])
def test_job_energies_over_k_chunks(o, v, cuda_dev):
    """Virtuals past one K chunk: a list of jobs with equal and distinct indices."""
    L = _system(o, v, 0.02)
    jobs = np.array([(v - 1, v - 1, v - 1), (v - 1, v - 1, 0), (v - 1, 3, 3), (v // 2, 2, 1), (5, 4, 0), (1, 1, 0)],
                    dtype=np.int32)
    ref = onp.job_energies(L, jobs.astype(np.int64)).sum()
    e = surrogate.energy_on_jobs(_dev(L, cuda_dev), jobs).item()
    assert abs(e - ref) <= 1e-12 * abs(ref)


@pytest.mark.parametrize("o,v,block", [(9, 7, None), (23, 6, None), (24, 7, (2, 7, 0, 2)), (12, 8, (3, 6, 3, 6))])
def test_lno_vjp_matches_oracle(o, v, block, cuda_dev):
    L = _system(o, v, 0.02)
    u = np.random.default_rng(1).standard_normal((max(1, o // 2), o))
    mat = u.T @ u
    e_ref, mb_ref, g_ref = onp.lno_energy_vjp(L, mat, 0.7, block=block)
    e, mb, g = triples.lno_energy_vjp(_dev(L, cuda_dev), torch.from_numpy(mat).to(cuda_dev), 0.7, block=block)
    assert abs(e.item() - e_ref) <= 1e-11 * abs(e_ref)
    assert np.linalg.norm(mb.cpu().numpy() - mb_ref) <= 1e-10 * np.linalg.norm(mb_ref)
    for k in KEYS:
        err = np.linalg.norm(g[k].cpu().numpy() - g_ref[k])
        assert err <= 1e-10 * np.linalg.norm(g_ref[k]) + 1e-15, (k, err)


@pytest.mark.parametrize("n", [1, 56, 220, 2024, 2300, 11480, 102340])
def test_job_energy_sum(n, cuda_dev):
    """The energy is the exact sum of the job energies at every size of the
    reduction (one CTA, several, the widest), to one rounding."""
    v = next(x for x in range(1, 200) if x * (x + 1) * (x + 2) // 6 >= n)
    L = _dev(_system(2, v, 0.0), cuda_dev)
    je = torch.empty(v * (v + 1) * (v + 2) // 6, dtype=torch.float64, device=cuda_dev)
    e = triples.energy(L, job_e=je).item()
    ref = math.fsum(je.cpu().tolist())
    assert abs(e - ref) <= 2.3e-16 * abs(ref)
