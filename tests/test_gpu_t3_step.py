"""GPU: ct_t3_step (foo' products formed from t3's cubes) against ct_t3_update
(foo' t3 formed as one GEMM) on amplitudes without any permutation symmetry, at
the smallest cubes, at odd and even nocc, on both sides of the staged cubes limit (nocc 20 / 22) and
with an element count that fills the grid unevenly.  Both are float64 sums of
the same terms: 1e-13 of the largest element, sums 1e-12 relative."""
import ctypes

import pytest
import torch

from pyscfad_b200 import native, triples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(1, 1), (1, 7), (2, 5), (3, 4), (7, 9), (8, 23), (16, 3), (20, 3), (21, 3), (22, 3)])
def test_step_equals_update(o, v, cuda_dev):
    g = torch.Generator(device=cuda_dev).manual_seed(o * 100 + v)
    kw = dict(dtype=torch.float64, device=cuda_dev, generator=g)
    mo = torch.cat([-0.3 - torch.rand(o, **kw), 0.1 + torch.rand(v, **kw)])
    foo = torch.randn((o, o), **kw)
    t3, t3c, t3x, tvv = (torch.randn((v, v, v, o, o, o), **kw) for _ in range(4))
    off = foo.clone()
    off.diagonal().zero_()
    too = torch.mm(off, t3.permute(3, 0, 1, 2, 4, 5).reshape(o, -1))
    new, ref = torch.empty_like(t3), torch.empty_like(t3)
    s0, s1 = (torch.zeros(2, dtype=torch.float64, device=cuda_dev) for _ in range(2))
    w = torch.empty(native.T3_STEP_WORK, dtype=torch.float64, device=cuda_dev)
    p = lambda *ts: [ctypes.c_void_p(t.data_ptr()) for t in ts]  # noqa: E731
    st = triples._stream(cuda_dev)
    native.check(native.lib().ct_t3_update(o, v, *p(mo, t3c, tvv, too, t3, t3x, ref), None, *p(s0), st))
    native.check(native.lib().ct_t3_step(o, v, *p(mo, foo, t3c, tvv, t3, t3x, new, s1, w), st))
    assert (new - ref).abs().max() <= 1e-13 * ref.abs().max()
    assert (s0 - s1).abs().max() <= 1e-12 * s0.abs().max()
    # the outputs must not alias what P3 reads at other elements
    assert native.lib().ct_t3_step(o, v, *p(mo, foo, t3c, tvv, t3, t3x, t3, s1, w), st) == -1
