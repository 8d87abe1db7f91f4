"""The sum of the job energies on both sides of the size from which its CTAs take
1024 threads: the exact sum of the job energies to one rounding."""
import math

import pytest
import torch

from pyscfad_b200 import synth, triples

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [183, 184])   # 1,038,220 and 1,055,240 jobs; the line lies at 2^20
def test_long_job_energy_sum(v, cuda_dev):
    L = synth.device_layouts(2, v, 2 * v, 3, device=cuda_dev)
    je = torch.empty(v * (v + 1) * (v + 2) // 6, dtype=torch.float64, device=cuda_dev)
    assert (je.numel() > 1 << 20) is (v == 184)
    e = triples.energy(L, job_e=je).item()
    ref = math.fsum(je.cpu().tolist())
    assert abs(e - ref) <= 2.3e-16 * abs(ref)
