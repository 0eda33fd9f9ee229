"""The y-operators on even and odd parts (jsd_parity.cuh) on the host: halves,
fragment order, extra row and column against the whole product in long double,
for every symmetry the kernel takes and Ny at the edges of its tiles (one row
beyond, one short, even and odd, the smallest and the largest). Compiles host
code with nvcc; no GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _nvcc():
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    return None


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not available")
def test_products_on_even_and_odd_parts(tmp_path):
    exe = tmp_path / "parity_check"
    subprocess.run([_nvcc(), "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(exe),
                    os.path.join(HERE, "host_kernels", "parity_check.cu")], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [ln.split() for ln in out if ln.strip()]
    assert len(rows) == 21 * 6
    # at most K roundings of products and sums, one of the operator and two of the parts
    for kind, m, k, err, plain in rows:
        assert float(err) < (int(k) + 3) * 2.0 ** -53 * 2, (kind, m, k, err)
