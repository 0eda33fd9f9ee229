"""The lane-pair half-split transform and the 9- and 16-point register DFTs
(jsd_fftsq.cuh) on the host, lanes emulated one after another through the
swizzled exchange buffer, against a direct DFT in long double. Compiles host
code with nvcc; no GPU."""
import os
import subprocess

import pytest

from test_fftsq_host import HERE, _nvcc


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not available")
def test_lane_pair_transforms_match_direct_dft(tmp_path):
    exe = tmp_path / "fftsq_pairs_check"
    subprocess.run([_nvcc(), "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(exe),
                    os.path.join(HERE, "host_kernels", "fftsq_pairs_check.cu")], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [ln.split() for ln in out if ln.strip()]
    assert {r[0] for r in rows} == {"pairs12", "pairs14", "pairs16", "dft9", "dft16"}
    for name, fwd, inv in rows:
        assert float(fwd) < 1e-14 and float(inv) < 1e-14, (name, fwd, inv)
