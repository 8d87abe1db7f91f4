"""The DF factor gradients where their sums run in several parts: repeated calls
give the same bits (the parts meet in a fixed order), and the values are the
oracle's to 1e-12 of each array's norm (test_gpu_df.py)."""
import numpy as np
import pytest
import torch

from oracle import df_np
from pyscfad_b200.cc import df

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v,naux", [(2, 37, 30), (5, 41, 64), (8, 60, 130), (3, 90, 257), (16, 40, 200)])
def test_factor_bars_repeat_bitwise(o, v, naux, cuda_dev):
    g = np.random.default_rng(o * v)
    n = o + v
    Loo, Lov = g.standard_normal((naux, o, o)), g.standard_normal((naux, o * v))
    Lvv = g.standard_normal((naux, v, v))
    Gvo, Gvv = g.standard_normal((v, o, o, o)), g.standard_normal((v, v, o, n))
    bars = {"vooo": torch.from_numpy(Gvo).to(cuda_dev), "vvop": torch.from_numpy(Gvv).to(cuda_dev)}
    first = df.df_factor_bar(bars, Loo, Lov, Lvv)
    for got, w in zip(first, df_np.factor_bar(Gvo, Gvv, Loo, Lov, Lvv, o, v)):
        assert np.linalg.norm(got.cpu().numpy() - w.reshape(got.shape)) <= 1e-12 * np.linalg.norm(w)
    for _ in range(10):
        for a, b in zip(first, df.df_factor_bar(bars, Loo, Lov, Lvv)):
            assert torch.equal(a, b)
