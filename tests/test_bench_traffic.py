"""bench.py multiplies DRAM bytes captured under ncu by times it measures: only as long as the kernels are those of the
capture."""
import json
import os
import shutil

import pytest

import bench
from helpers import ROOT


@pytest.fixture
def tree(tmp_path):
    """The captured figures and the kernel sources, with a digest that fits."""
    shutil.copytree(os.path.join(ROOT, "custom_op_benchmark_b200", "csrc"), tmp_path / "custom_op_benchmark_b200" / "csrc")
    shutil.copytree(os.path.join(ROOT, "profiles"), tmp_path / "profiles")
    path = tmp_path / "profiles" / "dram_traffic.json"
    figures = json.loads(path.read_text())
    for name, f in figures.items():
        if name != "_comment":
            f["digest"] = bench.code_digest(f["sources"], str(tmp_path))
    path.write_text(json.dumps(figures))
    return tmp_path


def test_figures_go_with_the_kernels_they_were_captured_on(tree):
    root, csrc = str(tree), tree / "custom_op_benchmark_b200" / "csrc"
    assert bench.traffic_for("attention_fwd", "rmat21_attention", root=root) > 1e9
    assert bench.traffic_for("attention_fwd", "rmat21_attention", scale=18, root=root) is None
    assert bench.traffic_for("attention_fwd", "zipf_attention", root=root) is None
    assert bench.traffic_for("carry_rows", "rmat21_attention", root=root) is None
    with open(csrc / "gk_group.cuh", "a") as f:
        f.write("\n// a comment\n")
    assert bench.traffic_for("attention_fwd", "rmat21_attention", root=root) > 1e9
    with open(csrc / "gk_group.cuh", "a") as f:
        f.write("constexpr int kAnother = 1;\n")
    assert bench.traffic_for("attention_fwd", "rmat21_attention", root=root) is None
    assert bench.traffic_for("attention_fwd_banded", "banded_attention", root=root) > 1e8
