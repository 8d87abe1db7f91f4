"""The LNO projections at the edges of their tile counts (nocc 16, 17, 32, 33,
48, 49) against the numpy oracle, and the mixed modes at one size per count.

Tolerances: the repository's (float64: energies 1e-11 relative, gradients 1e-10
of each gradient's norm; mixed: test_gpu_lno.MIXED_TOL / MIXED_GRAD_TOL)."""
import numpy as np
import pytest
import torch

from oracle import ccsd_t_np as onp
from pyscfad_b200 import synth, triples

pytestmark = pytest.mark.gpu


def _case(o, v, dev):
    L = synth.reference_layouts(synth.make_system(o, v, 3 * v, 9, fvo_sigma=0.02))
    u = np.random.default_rng(2).standard_normal((max(1, o // 3), o))
    D = {k: torch.from_numpy(np.ascontiguousarray(x)).to(dev) for k, x in L.items()}
    return L, D, u.T @ u


@pytest.mark.parametrize("o,v", [(16, 5), (17, 4), (32, 3), (33, 4), (48, 3), (49, 3)])
def test_projection_matches_oracle(o, v, cuda_dev):
    L, D, mat = _case(o, v, cuda_dev)
    e_ref, mb_ref, g_ref = onp.lno_energy_vjp(L, mat, 0.7)
    md = torch.from_numpy(mat).to(cuda_dev)
    e, mb, g = triples.lno_energy_vjp(D, md, 0.7)
    assert abs(e.item() - e_ref) <= 1e-11 * abs(e_ref)
    assert abs(triples.lno_energy(D, md).item() - e_ref) <= 1e-11 * abs(e_ref)
    assert np.linalg.norm(mb.cpu().numpy() - mb_ref) <= 1e-10 * np.linalg.norm(mb_ref)
    for k in triples.KEYS:
        err = np.linalg.norm(g[k].cpu().numpy() - g_ref[k])
        assert err <= 1e-10 * np.linalg.norm(g_ref[k]) + 1e-15, (k, err)


@pytest.mark.parametrize("mode,tol,gtol", [("tf32", 5e-5, 2e-3), ("bf16x3", 1e-5, 2e-4)])
@pytest.mark.parametrize("o,v", [(16, 6), (24, 5), (40, 4), (56, 3)])
def test_mixed_projection_matches_fp64(o, v, mode, tol, gtol, cuda_dev):
    _, D, mat = _case(o, v, cuda_dev)
    md = torch.from_numpy(mat).to(cuda_dev)
    e64, mb64, g64 = triples.lno_energy_vjp(D, md, 0.7)
    e, mb, g = triples.lno_energy_vjp(D, md, 0.7, mode=mode)
    assert abs(e.item() - e64.item()) <= tol * abs(e64.item())
    assert float(torch.linalg.norm(mb - mb64)) <= gtol * float(torch.linalg.norm(mb64))
    for k in ("t2T", "vooo", "vvop"):
        assert float(torch.linalg.norm(g[k] - g64[k])) <= gtol * float(torch.linalg.norm(g64[k])), k
