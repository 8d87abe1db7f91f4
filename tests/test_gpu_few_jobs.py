"""Energies over job lists at nocc 2-24 with 128 or more virtuals: few jobs take
the slot path (a job cut into many CTAs), more the shared-memory cube (one CTA
per job, which took 1.2 to 1.9 times as long on a few jobs of nocc=20/nvir=300).
Both against the numpy oracle, 1e-12 of the sum of the job energies' magnitudes
(the repository's float64 energy tolerance)."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import ccsd_t_np as onp
from pyscfad_b200 import native, surrogate

pytestmark = pytest.mark.gpu
EPILOGUE = 2   # profile kind: launched by the slot path only


def _layouts(o, v, seed):
    g = np.random.default_rng(seed)
    e = np.concatenate([np.sort(g.uniform(-2, -0.3, o)), np.sort(g.uniform(0.1, 3, v))])
    return dict(mo_energy=e, t1T=1e-2 * g.standard_normal((v, o)), t2T=1e-2 * g.standard_normal((v, v, o, o)),
                vooo=0.1 * g.standard_normal((v, o, o, o)), fvo=1e-2 * g.standard_normal((v, o)),
                vvop=0.1 * g.standard_normal((v, v, o, o + v)))


@pytest.mark.parametrize("o,v,njobs,slots", [(2, 200, 1, True), (4, 200, 110, True), (4, 200, 120, False),
                                             (3, 256, 320, True), (3, 256, 321, False), (17, 128, 3, True),
                                             (17, 128, 80, False), (8, 127, 3, False)])
def test_job_lists(o, v, njobs, slots, cuda_dev):
    L = _layouts(o, v, o + njobs)
    rng = np.random.default_rng(njobs)
    jobs = np.sort(rng.integers(0, v, (njobs, 3)), axis=1)[:, ::-1].astype(np.int32)
    jobs = np.unique(jobs, axis=0).copy()
    while len(jobs) < njobs:
        extra = np.sort(rng.integers(0, v, (njobs, 3)), axis=1)[:, ::-1].astype(np.int32)
        jobs = np.unique(np.concatenate([jobs, extra]), axis=0)[:njobs].copy()
    ref = onp.job_energies(L, jobs.astype(np.int64))
    D = {k: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_dev) for k, x in L.items()}
    native.check(native.lib().ct_profile_enable(1))
    try:
        e = surrogate.energy_on_jobs(D, jobs).item()
        tot, n = ctypes.c_double(0), ctypes.c_int(0)
        native.check(native.lib().ct_profile_read(EPILOGUE, ctypes.byref(tot), ctypes.byref(n)))
    finally:
        native.check(native.lib().ct_profile_enable(0))
    assert (n.value > 0) is slots
    assert abs(e - ref.sum()) <= 1e-12 * np.abs(ref).sum()
