"""float64 calls under CUDA graph capture once the workspace of their size exists:
an LNO VJP after an LNO energy of the same system (it allocates nothing of its
own).  A replay gives the values of a plain call: energies to 1e-13 relative,
gradients (atomic sums) to 1e-12 of their norm."""
import numpy as np
import pytest
import torch

from pyscfad_b200 import native, synth, triples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(7, 9), (26, 5)])
def test_lno_vjp_captured_after_an_energy(o, v, cuda_dev):
    L = {k: torch.from_numpy(np.ascontiguousarray(x)).to(cuda_dev)
         for k, x in synth.reference_layouts(synth.make_system(o, v, 3 * v, 3, fvo_sigma=0.02)).items()}
    mat = torch.eye(o, dtype=torch.float64, device=cuda_dev)
    mat[0, o - 1] = 0.25
    native.lib().ct_release_workspace()
    triples.lno_energy(L, mat)
    grads = {k: torch.zeros_like(x) for k, x in L.items()}
    mb = torch.zeros_like(mat)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        e, _, _ = triples.lno_energy_vjp(L, mat, 0.7, grads, mb)
    graph.replay()
    torch.cuda.synchronize()
    e_ref, mb_ref, g_ref = triples.lno_energy_vjp(L, mat, 0.7)
    assert abs(e.item() - e_ref.item()) <= 1e-13 * abs(e_ref.item())
    assert torch.linalg.norm(mb - mb_ref) <= 1e-12 * torch.linalg.norm(mb_ref)
    for k in triples.KEYS:
        assert torch.linalg.norm(grads[k] - g_ref[k]) <= 1e-12 * torch.linalg.norm(g_ref[k])
