"""The FP64 plan's own eigenbasis tables (symmetric_tables, jsd_parity.cuh) on the
host: exactly even and odd, even modes first, and consistent with each other: w0
and wN are D's wall rows times the new V, c0 and cN the new V^-1 times the even
part of the boundary columns of D^2, both against long double. Compiles host code with nvcc;
no GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from jax_spectral_dns._ops import operator_tables

HERE = os.path.dirname(os.path.abspath(__file__))
NAMES = ("D", "V", "Vinv", "lam", "sgn", "c0", "cN", "w0", "wN")
EPS, EPS_LD = 2.0 ** -53, 2.0 ** -64


def _nvcc():
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    return None


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if _nvcc() is None:
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("tables") / "tables_check"
    subprocess.run([_nvcc(), "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(exe),
                    os.path.join(HERE, "host_kernels", "tables_check.cu")], check=True, capture_output=True)
    return str(exe)


def _run(program, ny, tables):
    data = np.int32(ny).tobytes() + b"".join(np.ascontiguousarray(tables[k], dtype=np.float64).tobytes() for k in NAMES)
    out = subprocess.run([program], input=data, check=True, capture_output=True).stdout
    ok, n_even = np.frombuffer(out, dtype=np.int32, count=2)
    flat, got, at, n = np.frombuffer(out, dtype=np.float64, offset=8), {}, 0, ny - 2
    if ok:
        for k in NAMES:
            shape = (ny, ny) if k == "D" else (n, n) if k in ("V", "Vinv") else (n,)
            got[k] = flat[at: at + int(np.prod(shape))].reshape(shape)
            at += int(np.prod(shape))
    return bool(ok), int(n_even), got


@pytest.mark.parametrize("ny", [10, 17, 18, 33, 65, 98, 129, 145, 194])
def test_tables_belong_together(program, ny):
    t = operator_tables(ny)
    ok, n_even, g = _run(program, ny, {k: getattr(t, k) for k in NAMES})
    n, s = ny - 2, g["sgn"]
    assert ok and n_even == (n + 1) // 2 and np.array_equal(s, np.where(np.arange(n) < n_even, 1.0, -1.0))
    assert np.array_equal(g["D"], -g["D"][::-1, ::-1])
    assert np.array_equal(g["V"], s * g["V"][::-1]) and np.array_equal(g["Vinv"], s[:, None] * g["Vinv"][:, ::-1])
    assert np.array_equal(np.sort(g["lam"]), np.sort(t.lam))
    D, V, W = (g[k].astype(np.longdouble) for k in ("D", "V", "Vinv"))
    for name, row in (("w0", 0), ("wN", -1)):
        want, mag = D[row, 1:-1] @ V, np.abs(D[row, 1:-1]) @ np.abs(V)
        assert np.all(np.abs(g[name] - want) <= EPS * np.abs(want) + 2 * n * EPS_LD * mag), name
    # c0, cN: the even part of the caller's D^2 under the new V^-1; the caller's products are in 64 bits
    D2 = t.D2.astype(np.longdouble)
    D2 = (D2 + D2[::-1, ::-1]) / 2
    for name, col in (("c0", 0), ("cN", -1)):
        want = W @ D2[1:-1, col]
        mag = (np.abs(t.Vinv) + np.abs(t.Vinv[:, ::-1])) @ (np.abs(t.D) @ np.abs(t.D[:, col]))[1:-1]
        assert np.all(np.abs(g[name] - want) <= 4 * ny * EPS * mag), name
    assert np.array_equal(g["cN"], s * g["c0"]) and np.array_equal(g["wN"], -s * g["w0"])


def test_tables_without_definite_parity_are_left_alone(program):
    t = operator_tables(33)
    tables = {k: getattr(t, k).copy() for k in NAMES}
    tables["V"][3, 4] += 1e-6
    assert not _run(program, 33, tables)[0]
    tables = {k: getattr(t, k).copy() for k in NAMES}
    tables["D"][2, 2] = np.nan
    assert not _run(program, 33, tables)[0]
