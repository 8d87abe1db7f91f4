"""The float64 slot path's GEMMs (ct_pair.cu) against the numpy oracle, at the
edges of their tiles: every count of 8-row tiles in use, even and odd sizes
(16- and 8-byte copies), column groups of virtuals, arrays off a 16-byte
boundary, and term lists longer than one block of descriptors.

Tolerances: the repository's float64 ones (energies 1e-12 relative, gradients
1e-10 of each gradient's norm)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import ccsd_t_np as onp
from pyscfad_b200 import native, surrogate, synth, triples

pytestmark = pytest.mark.gpu
KEYS = triples.KEYS


def _system(o, v, fvo=0.02, seed=7):
    return synth.reference_layouts(synth.make_system(o, v, 3 * v, seed, fvo_sigma=fvo))


def _dev(L, dev, shift=0):
    """The layouts on the device, each `shift` doubles past an aligned address."""
    out = {}
    for k, x in L.items():
        x = np.ascontiguousarray(x)
        buf = torch.empty(x.size + shift, dtype=torch.float64, device=dev)
        out[k] = buf[shift:].view(x.shape).copy_(torch.from_numpy(x))
    return out


def _close(g, g_ref):
    for k in KEYS:
        err = np.linalg.norm(g[k].cpu().numpy() - g_ref[k])
        assert err <= 1e-10 * np.linalg.norm(g_ref[k]) + 1e-15, (k, err)


@pytest.mark.parametrize("o,v,shift", [(1, 4, 0), (25, 3, 0), (26, 8, 0), (26, 8, 1), (32, 6, 0), (33, 4, 0), (34, 5, 0),
                                       (40, 4, 0), (41, 3, 0), (48, 6, 0), (49, 3, 0), (56, 4, 0), (57, 3, 0),
                                       (64, 4, 0), (30, 2, 0)])
def test_vjp_matches_oracle(o, v, shift, cuda_dev):
    L = _system(o, v)
    e_ref, g_ref = onp.energy_vjp(L, 1.0)
    D = _dev(L, cuda_dev, shift)
    e, g = triples.energy_vjp(D, 2.0)
    assert abs(e.item() - e_ref) <= 1e-12 * abs(e_ref) + 1e-14
    assert abs(triples.energy(D).item() - e_ref) <= 1e-12 * abs(e_ref) + 1e-14
    _close(g, g_ref)


@pytest.mark.parametrize("o,v", [(25, 66), (26, 130), (40, 64)])
def test_block_over_long_lists(o, v, cuda_dev, monkeypatch):
    """Two slab pairs with every smaller index: several column groups of
    virtuals, several K stages, and groups of more terms than a descriptor block."""
    L = _system(o, v)
    jobs = np.array([(a, b, c) for a in (v - 2, v - 1) for b in range(v - 2, a + 1) for c in range(b + 1)])
    monkeypatch.setattr(onp, "sorted_jobs", lambda *a: jobs)
    e_ref, g_ref = onp.energy_vjp(L, 1.0)
    D = _dev(L, cuda_dev)
    g = {k: torch.zeros_like(x) for k, x in D.items()}
    e = torch.zeros((), dtype=torch.float64, device=cuda_dev)
    ptr = lambda d: [ctypes.c_void_p(d[k].data_ptr()) for k in KEYS]  # noqa: E731
    prob, grads = native.CtProblem(o, v, *ptr(D)), native.CtGrads(*ptr(g))
    native.check(native.lib().ct_energy_vjp_block(ctypes.byref(prob), 0, 2.0, ctypes.byref(grads), v - 2, v, v - 2, v,
                                                  ctypes.c_void_p(e.data_ptr()), None))
    torch.cuda.synchronize()
    assert abs(e.item() - e_ref) <= 1e-12 * abs(e_ref)
    _close(g, g_ref)


@pytest.mark.parametrize("o,v", [(25, 17), (31, 33), (48, 16), (63, 18)])
def test_job_energies(o, v, cuda_dev):
    L = _system(o, v)
    jobs = np.array([(v - 1, v - 1, v - 1), (v - 1, v - 1, 0), (v - 1, 3, 3), (v // 2, 2, 1), (5, 4, 0)], dtype=np.int32)
    ref = onp.job_energies(L, jobs.astype(np.int64)).sum()
    assert abs(surrogate.energy_on_jobs(_dev(L, cuda_dev), jobs).item() - ref) <= 1e-12 * abs(ref)
