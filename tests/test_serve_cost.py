"""The serving loops size their waves by set_cost_us (pl_serve_plan.cuh): its
figure at each bin's largest k is the time of a set at the rate that the
autotuner measured for the kernel that runs there (tuning.json), within 10%.
Needs nvcc (host code only), no GPU."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_set_costs_are_the_measured_rates(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc absent")
    with open(os.path.join(ROOT, "paralanczos_b200", "tuning.json")) as f:
        bins = {b["kmax"]: 1e6 / b["sets_per_s"] for b in json.load(f)["bins"].values()}
    src = tmp_path / "cost.cu"
    src.write_text('#include <stdio.h>\n#include "%s/paralanczos_b200/csrc/pl_serve_plan.cuh"\nint main() {\n%s}\n' % (
        ROOT, "".join(f'  printf("{k} %.9g\\n", pl::serve::set_cost_us({k}));\n' for k in bins)))
    exe = tmp_path / "cost"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", str(src), "-o", str(exe)], check=True,
                   capture_output=True, text=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    got = {int(k): float(v) for k, v in (line.split() for line in out.splitlines())}
    assert set(got) == set(bins)
    for k, want in bins.items():
        assert abs(got[k] - want) <= 0.1 * want, (k, got[k], want)
