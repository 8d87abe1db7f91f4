"""bench.py's roofline: the flops of the float64 kernel kinds follow the path a
size takes (one kernel per job at nocc 2-24), and the table of DRAM bytes names
kernels that exist."""
import glob
import json
import os
import re

import pytest

import bench
from conftest import ROOT


@pytest.mark.parametrize("o,v", [(2, 9), (16, 120), (24, 60)])
def test_job_kernel_counts_its_products(o, v):
    w, vb, ob = 12 * o ** 3 * (v + o), 12 * o ** 3 * v, 12 * o ** 4
    assert bench.roofline_units(0, "fp64", o, v) == ("tensor", w + vb + 2 * ob, "TFLOP/s")


@pytest.mark.parametrize("o", [1, 25, 48])
def test_slot_path_w_build(o):
    assert bench.roofline_units(0, "fp64", o, 100)[1] == 12 * o ** 3 * (100 + o)


def test_traffic_table_names_present_kernels():
    src = "".join(open(p).read() for p in glob.glob(os.path.join(ROOT, "pyscfad_b200", "csrc", "*.cu")))
    limit = int(re.search(r"kCubeMaxO = (\d+)", open(os.path.join(ROOT, "pyscfad_b200", "csrc", "ct_internal.h")).read())[1])
    assert bench.CUBE_MAX_O == limit
    table = json.load(open(os.path.join(ROOT, "profiles", "roofline_traffic.json")))
    for mode in ("fp64", "tf32", "bf16x3"):
        for kind, e in table[mode].items():
            name = re.search(r"(?:\w+::)?(\w+_kernel)", e["kernel"])[1]
            assert re.search(r"\b%s\b" % name, src), (mode, kind, name)
    # the slot path has no separate vooo pass
    assert "1" not in table["fp64"]
