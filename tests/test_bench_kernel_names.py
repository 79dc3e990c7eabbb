"""The kernel that the bench names for a sloppy-hop tile is the one that the library launches for it (CPU)."""
import importlib.util
import os
import re

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("precision,tile,kernel", [
    ("single", (1, 64, 0), "hop_f32_kernel"), ("single", (1, 256, 0), "hop_f32_kernel"),
    ("single", (2, 128, 0), "hop_mrhs_kernel"), ("single", (1, 128, 12), "hop_mu4_kernel"),
    ("double", (1, 256, 0), "hop_mrhs_kernel"), ("half", (1, 64, 0), "hop_mrhs_kernel"),
    ("half", (2, 64, 0), "hop_pair_kernel"), ("half", (2, 64, 11), "hop_pair_hp_kernel"),
    ("half", (1, 128, 12), "hop_mu4_kernel")])
def test_names_follow_the_launcher(bench, precision, tile, kernel):
    assert bench.hop_kernel_name(precision, tile) == kernel
    launcher = open(os.path.join(ROOT, "qkxtm_mpi_b200", "csrc", "mixed.cu")).read()
    assert re.search(rf"\b{kernel}<", launcher)
