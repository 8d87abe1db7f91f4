"""The tensor-core t2-bar and vooo-bar GEMMs at short and ragged term lists
(one, two or four terms per stage by nocc) against the float64 path.

Tolerances: the repository's mixed-mode ones for gradients (test_gpu_mixed.TOL)."""
import numpy as np
import pytest
import torch

from pyscfad_b200 import synth, triples

pytestmark = pytest.mark.gpu
GRAD_TOL = {"tf32": 2e-3, "bf16x3": 2e-4}


@pytest.mark.parametrize("mode", ["tf32", "bf16x3"])
@pytest.mark.parametrize("o,v", [(8, 2), (8, 5), (8, 13), (16, 3), (16, 10), (24, 6), (40, 5)])
def test_bars_match_fp64(o, v, mode, cuda_dev):
    L = synth.reference_layouts(synth.make_system(o, v, 3 * v, 11, fvo_sigma=0.02))
    D = {k: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_dev) for k, x in L.items()}
    _, g64 = triples.energy_vjp(D, 2.0)
    _, g = triples.energy_vjp(D, 2.0, mode=mode)
    for k in ("t2T", "vooo", "vvop"):
        err = float(torch.linalg.norm(g[k] - g64[k]))
        assert err <= GRAD_TOL[mode] * float(torch.linalg.norm(g64[k])), (k, err)


@pytest.mark.parametrize("mode", ["tf32", "bf16x3"])
@pytest.mark.parametrize("o,v", [(32, 3), (32, 8), (8, 30), (16, 21), (48, 4)])
def test_bars_match_fp64_by_terms_per_stage(o, v, mode, cuda_dev):
    """nocc 32 (two terms of vooo-bar, one of t2-bar a stage), eight and four terms
    a stage over lists that do not divide by them, one term at nocc 48."""
    test_bars_match_fp64(o, v, mode, cuda_dev)
