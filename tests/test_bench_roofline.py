"""bench.py's roofline entry names the kernels that the plan's choices run and
divides the operations that they execute by the peak; a kernel without a profile has no traffic figure. No GPU."""
import os

import pytest

import bench
from conftest import REPO

MODES = (129, 129, 129)
PEAKS = {"hbm_gbs": 6538.0, "bf16_tflops": 1650.0}
N = 2 * 129 * 129


def _choices(even_odd=True, eig=(0, 0), xmid=1, split=1):
    return {"eig_kernel": list(eig), "even_odd": [even_odd] * 3, "split_kernel": split, "xmid_variant": xmid}


def _line(dom, form, choices, work, us):
    kernels = {dom: {"ms": us / 1e3, "launches": 1, "work": work}, "other": {"ms": us / 1e3, "launches": 1, "work": 1.0}}
    return bench.roofline_line(dom, kernels, form, choices, MODES, PEAKS, "measured", (35.4, 15.6))


def test_products_on_even_and_odd_parts_count_what_runs():
    # y-derivatives of two fields in 67 us: two halves of 65 x 64 (and 64 x 65) each
    work = 2 * 2.0 * (65 * 64 + 64 * 65) * N
    out = _line("gemm", "fp64", _choices(), work, 67.0)
    assert out["kernel"].startswith("k_parity (") and out["unit"] == "TFLOP/s"
    assert out["frac"] == pytest.approx(work / 67e-6 / 1e12 / 35.4) and out["frac"] < 1
    assert out["whole_operator_equivalent_tflops"] == pytest.approx(2 * out["achieved"], rel=0.02)
    assert out["share_of_kernel_time"] == 0.5


@pytest.mark.parametrize("dom,form,choices,name", [
    ("gemm", "fp64", _choices(even_odd=False), "k_dgemm"),
    ("gemm", "fp64", _choices(eig=(1, 0)), "k_parity / k_dgemm / k_oz8_gemm"),
    ("gemm", "mixed", _choices(False, (1, 1), 0), "k_oz8_gemm"),
    ("gemm", "mixed", _choices(False, (0, 1), 0), "k_dgemm + k_oz8_gemm"),
    ("gemm", "mixed", _choices(False, (0, 0), 0), "k_dgemm"),
    ("sgemm", "mixed", _choices(False, (1, 1), 0), "k_tc05_split"),
    ("sgemm", "mixed", _choices(False, (1, 1), 0, 0), "k_sgemm3"),
    ("xmid", "fp64", _choices(xmid=0), "k_xmid_park"), ("xmid", "fp64", _choices(xmid=1), "k_xmid_park"),
    ("xmid", "fp64", _choices(xmid=2), "k_xmid"), ("xmid", "mixed", _choices(xmid=0), "k_xmid_sq"),
    ("xmid", "mixed", _choices(xmid=1), "k_xmid_h2"), ("zinv", "fp64", _choices(), "k_zinv_staged"),
    ("zinv", "mixed", _choices(), "k_zinv_staged"), ("zfwd", "fp64", _choices(), "k_zfwd_sq"),
    ("eigen", "fp64", _choices(), "k_eigen_update")])
def test_names_limits_and_traffic_are_the_running_kernels(dom, form, choices, name):
    out = _line(dom, form, choices, 1e8, 100.0)
    stem = bench.kernel_of(dom, form, choices)
    assert out["kernel"].split(" (")[0] == name and (stem is None) == ("+" in name or "/" in name)
    profile = os.path.join(REPO, "profiles", f"{stem}_channel_128x129x128.md")
    if out["traffic"] is not None:
        assert os.path.exists(profile) and stem in out["traffic_source"]
    if not os.path.exists(profile):
        assert out["traffic"] is None
    assert ("limiter" in out) == (stem in ("k_xmid_sq", "k_xmid_park"))
    if "limiter" in out:
        assert os.path.exists(profile)
