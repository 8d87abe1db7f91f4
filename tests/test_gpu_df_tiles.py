"""The DF kernels in both tile builds (64 and 128 rows) and the sums in parts,
at sizes that are no multiples of the tiles, with K below one step and at single
elements, against the oracle at the tolerance of test_gpu_df.py (1e-12 of each
array's norm)."""
import numpy as np
import pytest
import torch

from oracle import df_np
from pyscfad_b200.cc import df

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v,naux", [(1, 1, 1), (5, 9, 3), (2, 33, 16), (8, 60, 70), (7, 61, 37), (3, 130, 17),
                                      (9, 24, 300)])
def test_products_match_oracle(o, v, naux, cuda_dev):
    g = np.random.default_rng(naux)
    n = o + v
    Loo, Lov, Lvv = g.standard_normal((naux, o * o)), g.standard_normal((naux, o * v)), g.standard_normal((naux, v, v))
    e = np.linspace(-1.0, 1.0, n)
    L = df.df_layouts(np.zeros((o, v)), np.zeros((o, o, v, v)), e, np.diag(e), Loo, Lov, Lvv, device=cuda_dev)
    Gvo, Gvv = g.standard_normal((v, o, o, o)), g.standard_normal((v, v, o, n))
    bars = df.df_factor_bar({"vooo": torch.from_numpy(Gvo).to(cuda_dev), "vvop": torch.from_numpy(Gvv).to(cuda_dev)},
                            Loo, Lov, Lvv)
    got = [L["vooo"], L["vvop"], *bars]
    want = [*df_np.vooo_vvop(Loo, Lov, Lvv, o, v), *df_np.factor_bar(Gvo, Gvv, Loo, Lov, Lvv, o, v)]
    for a, b in zip(got, want):
        assert np.linalg.norm(a.cpu().numpy() - b.reshape(tuple(a.shape))) <= 1e-12 * np.linalg.norm(b)
