"""The shared-memory cube path (ct_cube.cu) where a job's F1 sum takes several K
chunks and its columns one, two or three passes, against the numpy oracle, and
the t2-bar / vooo-bar GEMMs of both float64 paths on parts of more terms than one
block of descriptors, against the same system in short waves.

``launch_plan`` restates the launch rule of ct_cube.cu, so that a size that no
longer reaches several chunks fails here.  Tolerances: the repository's float64
ones (energies 1e-12 relative, gradients 1e-10 of each gradient's norm against
the oracle); 1e-12 of the norm between two orders of the same sums."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import ccsd_t_np as onp
from pyscfad_b200 import native, surrogate, synth, triples

KEYS = triples.KEYS
BUILDS = {1: (1, 2, 32, 16), 2: (2, 2, 128, 5), 3: (3, 3, 192, 3), 4: (4, 4, 256, 2), 5: (5, 3, 256, 2),
          6: (6, 3, 512, 1)}   # 8-row tiles, 8-column tiles, threads, CTAs per SM


def _strides(o):
    """Strides (j, i) of the padded cube: least bank conflicts, then least padding."""
    best = None
    for pj in range(4):
        for pi in range(8):
            j = o + pj
            s, cost = (o * j + pi, j, 1), 0
            for x in range(3):
                for y in range(3):
                    if x != y:
                        banks = [(u * s[x] + w * s[y]) % 16 for u in range(4) for w in range(4)]
                        cost += max(banks.count(b) for b in banks)
            if best is None or (cost, pj, pi) < best[:3]:
                best = (cost, pj, pi, j, s[0])
    return best[3:]


def launch_plan(o, v, vjp):
    """(column passes, K chunks) of the job kernel."""
    mt, nt, threads, ctas = BUILDS[(o + 3) // 4]
    if o == 20 and vjp:
        mt, nt, threads, ctas = 5, 2, 512, 1
    groups = -(-(-(-o * o // 8)) // nt)
    passes = -(-groups // (threads // 32))
    warps = -(-groups // passes)
    _, si = _strides(o)
    cube = (o * si + 1) & ~1
    part = max(o * (o + 1) * (o + 2) // 6, 6 * warps * 32) if vjp else 0
    room = (228 * 1024 // ctas - 2048) // 8 - cube - part - 7 * o
    cap = max(32, min(128, (room // (16 * mt) - 4) // 16 * 16))
    return passes, -(-v // cap)


@pytest.mark.parametrize("o", range(2, 25))
def test_shared_memory_fits(o):
    """Every size the cube path takes stays within an SM's 227 KB."""
    for vjp in (False, True):
        mt = 5 if o == 20 and vjp else BUILDS[(o + 3) // 4][0]
        _, si = _strides(o)
        for v in (1, 31, 64, 97, 112, 127, 128, 129, 300, 1024):
            passes, chunks = launch_plan(o, v, vjp)
            kc = max(32, -(-(-(-v // chunks)) // 16) * 16)
            part = max(o * (o + 1) * (o + 2) // 6, 6 * 16 * 32) if vjp else 0
            stage = max(16 * mt * (kc + 4), 12 * o * (o | 1))
            assert 8 * ((o * si + 2) + stage + part + 7 * o) + 384 <= 232448


def _layouts(o, v, seed):
    g = np.random.default_rng(seed)
    e = np.concatenate([np.sort(g.uniform(-2, -0.3, o)), np.sort(g.uniform(0.1, 3, v))])
    return dict(mo_energy=e, t1T=1e-2 * g.standard_normal((v, o)), t2T=1e-2 * g.standard_normal((v, v, o, o)),
                vooo=0.1 * g.standard_normal((v, o, o, o)), fvo=1e-2 * g.standard_normal((v, o)),
                vvop=0.1 * g.standard_normal((v, v, o, o + v)))


def _dev(L, dev):
    return {k: torch.from_numpy(np.ascontiguousarray(x)).to(dev) for k, x in L.items()}


# last chunks of 1, 2, 3, 15 and a full number of virtuals; nvir >= 128 needs the
# jobs of more than half the SMs to stay on this path
@pytest.mark.gpu
@pytest.mark.parametrize("o,v,njobs,passes", [(2, 81, 9, 1), (4, 127, 9, 1), (10, 129, 90, 1), (16, 130, 90, 1),
                                              (17, 97, 9, 2), (18, 82, 9, 2), (19, 95, 9, 2), (20, 65, 9, 3),
                                              (20, 127, 9, 3), (21, 131, 90, 2), (23, 129, 90, 2)])
def test_job_energies(o, v, njobs, passes, cuda_dev):
    plan = launch_plan(o, v, False)
    assert plan[0] == passes and plan[1] > 1
    L = _layouts(o, v, o)
    rng = np.random.default_rng(v)
    jobs = np.sort(rng.integers(0, v, (4 * njobs, 3)), axis=1)[:, ::-1]
    jobs = np.concatenate([[(v - 1, v - 1, v - 1), (v - 1, v - 1, 0), (v - 1, 3, 3)], jobs])
    jobs = np.unique(jobs, axis=0)[-njobs:].astype(np.int32).copy()
    ref = onp.job_energies(L, jobs.astype(np.int64))
    D = _dev(L, cuda_dev)
    native.check(native.lib().ct_profile_enable(1))
    try:
        e = surrogate.energy_on_jobs(D, jobs).item()
        tot, n = ctypes.c_double(0), ctypes.c_int(0)
        native.check(native.lib().ct_profile_read(2, ctypes.byref(tot), ctypes.byref(n)))
    finally:
        native.check(native.lib().ct_profile_enable(0))
    assert n.value == 0   # no slot-path epilogue
    assert abs(e - ref.sum()) <= 1e-12 * np.abs(ref).sum()


def _block(D, o, v, slab):
    g = {k: torch.zeros_like(x) for k, x in D.items()}
    e = torch.zeros((), dtype=torch.float64, device=D["t1T"].device)
    ptr = lambda d: [ctypes.c_void_p(d[k].data_ptr()) for k in KEYS]  # noqa: E731
    prob, grads = native.CtProblem(o, v, *ptr(D)), native.CtGrads(*ptr(g))
    native.check(native.lib().ct_energy_vjp_block(ctypes.byref(prob), 0, 2.0, ctypes.byref(grads), v - slab, v,
                                                  v - slab, v, ctypes.c_void_p(e.data_ptr()), None))
    torch.cuda.synchronize()
    return e.item(), g


@pytest.mark.gpu
@pytest.mark.parametrize("o,v", [(3, 67), (8, 115), (17, 83), (18, 66), (19, 65), (20, 131), (24, 113)])
def test_block_vjp(o, v, cuda_dev, monkeypatch):
    assert launch_plan(o, v, True)[1] > 1
    L = _layouts(o, v, v)
    jobs = np.array([(v - 1, v - 1, c) for c in range(v)])
    monkeypatch.setattr(onp, "sorted_jobs", lambda *a: jobs)
    e_ref, g_ref = onp.energy_vjp(L, 1.0)
    scale = np.abs(onp.job_energies(L, jobs)).sum()
    e, g = _block(_dev(L, cuda_dev), o, v, 1)
    assert abs(e - e_ref) <= 1e-12 * scale
    for k in KEYS:
        err = np.linalg.norm(g[k].cpu().numpy() - g_ref[k])
        assert err <= 1e-10 * np.linalg.norm(g_ref[k]) + 1e-15, (k, err)


@pytest.mark.gpu
@pytest.mark.parametrize("o,v,block", [(23, 52, 128), (25, 50, 64)])
def test_parts_longer_than_a_descriptor_block(o, v, block, cuda_dev, monkeypatch):
    """One wave of every job: parts of more terms than a block of descriptors
    (128 on the cube path, 64 on the slot path), against waves of 888 jobs."""
    njobs = v * (v + 1) * (v + 2) // 6
    tile = 64 if o <= 24 else 128
    assert 6 * njobs * (-(-v // 64)) * (-(-o * o // tile)) // (64 * 148) > block
    L = synth.device_layouts(o, v, 3 * v, 5, device=cuda_dev, fvo_sigma=0.02)
    out = {}
    try:
        for waves in (888, njobs):
            native.lib().ct_release_workspace()
            monkeypatch.setenv("CTB_MAX_WAVE", str(waves))
            out[waves] = triples.energy_vjp(L, 2.0)
            torch.cuda.synchronize()
    finally:
        monkeypatch.delenv("CTB_MAX_WAVE")
        native.lib().ct_release_workspace()
    (e0, g0), (e1, g1) = out[888], out[njobs]
    assert abs(e0.item() - e1.item()) <= 1e-13 * abs(e0.item())
    for k in KEYS:
        assert torch.linalg.norm(g1[k] - g0[k]) <= 1e-12 * torch.linalg.norm(g0[k]), k
