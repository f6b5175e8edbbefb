"""A packed binary32x2 product whose lanes go into scalar sums and differences
rounds every lane as the scalar product and the scalar sum do, in each of the
forms that the agent kernels use (tests/probes/packed_products.cu, the host's
arithmetic against the device's on 2 M lanes a form)."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

FORMS = ["sensor position", "sin/cos reduction", "bilinear interpolation", "jitter hash argument", "fraction"]


def test_packed_products_into_scalar_sums_round_twice(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "packed_products"
    # the library's own arithmetic flags
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "probes", "packed_products.cu")], check=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    lines = [line.split() for line in out.splitlines()]
    assert [int(k) for _, k, _, _ in lines] == list(range(len(FORMS)))
    for _, k, bad, lanes in lines:
        assert int(lanes) == 1 << 21 and int(bad) == 0, f"{FORMS[int(k)]}: {bad} of {lanes} lanes differ"
